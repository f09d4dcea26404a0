"""The host-side choices of grids for the decode kernels (no GPU needed): every choice must be one
that the kernels accept, whatever sizes a configuration brings."""

import itertools

from tokamak_b200.csrc import ops


def test_decode_splits_stay_in_one_wave_and_keep_the_warps_level():
    for n_items, hkv, kv_len in itertools.product((1, 2, 3, 4, 7, 8, 16, 37, 64, 300), (1, 2, 5, 8, 16),
                                                  (1, 15, 16, 17, 100, 1024, 4096, 40000, 131072)):
        s = ops.decode_splits(n_items, hkv, kv_len)
        assert 1 <= s <= 128
        tiles = -(-kv_len // 16)
        if s > 1:
            assert n_items * hkv * s <= 444                      # one wave: three blocks of two stages per SM
            per_split = -(-tiles // s)
            assert per_split >= 8                                # a block has enough to stream
            assert s * per_split >= tiles
    # the measured cases
    assert ops.decode_splits(8, 8, 4096) == 6            # 384 blocks: two stages, three to an SM
    assert ops.decode_splits(16, 8, 4096) == 3
    assert ops.decode_splits(1, 8, 4096) == 32           # 256 blocks: three stages, two to an SM
    assert ops.decode_splits(32, 8, 4096) == 1
    assert ops.decode_splits(64, 8, 4096) == 1


def test_short_contexts_take_the_split_decode_kernel(monkeypatch):
    device = "cuda:0"
    monkeypatch.setitem(ops._SM_COUNT, device, 148)
    monkeypatch.setattr(ops, "DECODE_ATTENTION", "auto")
    uses = lambda n, hkv, kv: ops.decode_uses_balanced(device, n, hkv, kv)
    # (pairs, key bucket) at the edges of the rule: 296 pairs, 444 pairs, buckets of 512 and 2,048
    assert [uses(37, 8, kv) for kv in (256, 2048, 4096)] == [False, False, False]
    assert [uses(38, 8, kv) for kv in (256, 2048, 4096)] == [False, False, True]
    assert [uses(55, 8, kv) for kv in (512, 2048, 4096)] == [False, False, True]
    assert [uses(56, 8, kv) for kv in (256, 512, 1024)] == [False, False, True]
    assert uses(1025, 8, 4096) is False and uses(1024, 1, 512) is False
    # rounds of 444 pairs three quarters full (two: from 666 on, three: 999) and not; heads of 64
    assert [uses(n, 8, 1024) for n in (64, 83, 84, 96, 111, 112, 124, 125, 128, 256)] == [True, True, False, False, False, True, True,
                                                                                          False, False, False]
    assert [uses(n, 8, 2048) for n in (96, 128)] == [False, False] and [uses(n, 8, 4096) for n in (96, 128)] == [True, True]
    assert [ops.decode_uses_balanced(device, 64, 8, kv, 64) for kv in (512, 2048, 4096)] == [False, False, True]


def test_swapped_gemm_plan_is_one_cluster_of_at_most_eight():
    for n_out, k, tokens in itertools.product((128, 1000, 4096, 6144, 24576, 34816, 151936), (64, 320, 1024, 4096, 17408),
                                              (1, 8, 16, 17, 64)):
        splits, stages, cluster = ops.swapped_gemm_plan(n_out, k, tokens)
        assert 1 <= splits <= 8 and cluster == splits
        assert stages in (3, 4)
        assert splits <= max(1, -(-k // 64))                      # no split without a k block
    # the shapes of the Qwen3-8B decode step at batch 8: q|k|v, output, gate/up, down, head
    assert ops.swapped_gemm_plan(6144, 4096, 8) == (8, 4, 8)
    assert ops.swapped_gemm_plan(4096, 4096, 8) == (8, 4, 8)
    assert ops.swapped_gemm_plan(24576, 4096, 8) == (2, 4, 2)
    assert ops.swapped_gemm_plan(4096, 12288, 8) == (8, 4, 8)
    assert ops.swapped_gemm_plan(151936, 4096, 8) == (1, 4, 1)
    # the splits, and with them the order of a token's sums, follow from the weight alone
    for n_out, k in itertools.product((128, 1000, 4096, 24576), (64, 320, 1024, 1536, 4096)):
        assert len({ops.swapped_gemm_plan(n_out, k, tokens)[::2] for tokens in (1, 2, 7, 8, 9, 16, 17, 33, 64)}) == 1
    # larger token tiles have larger stages: four of them only where two blocks per SM are enough
    assert ops.swapped_gemm_plan(151936, 4096, 64)[1] == 3
    assert ops.swapped_gemm_plan(4096, 4096, 64)[1] == 4


def test_pair_gemm_is_for_grids_that_fill_the_gpu():
    assert ops.pair_gemm_takes(2048, 4096, 4096)
    assert not ops.pair_gemm_takes(256, 4096, 4096)               # 16 tiles: the library is faster
    assert not ops.pair_gemm_takes(2048, 4096, 4100)              # inner size no multiple of 8


def test_sampling_refuses_sizes_its_histograms_cannot_hold():
    import pytest
    ops._sampling_takes(64, 151936)
    ops._sampling_takes(ops.SAMPLING_MAX_ROWS, ops.SAMPLING_MAX_VOCAB)
    with pytest.raises(ops.KernelError, match="sampling kernel takes"):
        ops._sampling_takes(1, ops.SAMPLING_MAX_VOCAB + 1)
    with pytest.raises(ops.KernelError, match="sampling kernel takes"):
        ops._sampling_takes(ops.SAMPLING_MAX_ROWS + 1, 1000)


def test_kernels_have_their_tensor_memory_before_anything_can_wait_for_them():
    """A block that lets later kernels begin (or waits for earlier ones) before its tensor memory is its own could find it
    taken by a block that waits for this one.  A block of the product chain, which fills an SM's shared memory and so is
    alone there, allocates before it waits; all others before they let anything begin."""
    from pathlib import Path
    csrc = Path(ops.__file__).resolve().parent
    for name, before in (("attention_prefill_tc", "pdl_trigger();"), ("gemm_pair_tcgen05", "pdl_trigger();"),
                         ("moe_stream", "pdl_trigger();"), ("gemm_tcgen05", "pdl_trigger();"), ("gemm_chain", "pdl_wait();")):
        text = (csrc / f"{name}.cu").read_text()
        assert text.count("tcgen05.alloc.") == 1, name
        kernel = text[text.index("__global__"):]
        assert kernel.index("tcgen05.alloc.") < kernel.index(before), name


def test_products_of_a_few_hundred_tokens_and_latent_prompts_have_their_tensor_memory_first():
    """The same for the product with the tokens on the N side and for prompts over a latent cache."""
    from pathlib import Path
    csrc = Path(ops.__file__).resolve().parent
    for name in ("gemm_tokens_tcgen05.cu", "latent_prefill.cuh"):
        text = (csrc / name).read_text()
        assert text.count("tcgen05.alloc.") == 1, name
        kernel = text[text.index("__global__"):]
        assert kernel.index("tcgen05.alloc.") < kernel.index("pdl_trigger();"), name


def test_the_experts_second_product_begins_behind_the_router():
    """It reads the router's choice before it waits for the first product.  That is sound because a block of the first lets it begin
    only once the first's own wait, for the router, is over; results alone would hardly show the race."""
    from pathlib import Path
    text = (Path(ops.__file__).resolve().parent / "moe_stream.cu").read_text()
    kernel = text[text.index("__global__"):]
    wait, trigger = kernel.index("if (!p.choice_is_there) pdl_wait();"), kernel.index("pdl_trigger();")
    assert kernel.index("tcgen05.alloc.") < wait < trigger < kernel.index("p.chosen + i")
    assert kernel.count("pdl_trigger();") == 1 and "__ldcg(p.chosen" in kernel and "p.chosen[" not in kernel


def test_the_float32_products_tile_follows_the_devices_sms():
    """Products and the tiles they were fastest with on 148 SMs (16, 32 and 64 rows), and the same rule on other counts: a
    block an SM at most for the lowest tile, two for the highest."""
    from tokamak_b200.csrc.lib import library
    tile = library().tk_gemm_f32_tile
    assert [tile(m, n, 1, 148) for m, n in ((254, 6144), (254, 1024), (100, 1024), (40, 4096), (16, 6144), (1, 151936))] == [3, 2, 1, 2, 1, 1]
    assert [tile(100, 1024, 1, sms) for sms in (20, 56, 111, 112, 148)] == [2, 2, 2, 1, 1]
    assert [tile(254, 6144, batch, sms) for batch, sms in ((1, 192), (1, 193), (2, 193), (2, 385))] == [3, 2, 3, 2]
    assert [tile(100, 1024, 1, sms) for sms in (16, 17)] == [3, 2]


def test_the_smallest_steps_of_small_experts_take_the_cuda_cores():
    """On both sides of every measured edge: pairs, and weights over all pairs."""
    takes = lambda n, per, width, ff: ops.moe_small_is_better(n, per, width, ff)
    assert [takes(n, 3, 264, 320) for n in (1, 2, 3, 4, 8, 21)] == [True, True, True, False, False, False]
    assert [takes(n, 2, 512, 256) for n in (1, 4, 5, 6, 32)] == [True, True, True, False, False]
    assert [takes(n, 2, 512, 512) for n in (1, 3, 4, 5, 6)] == [True, True, True, True, False]
    assert [takes(n, 4, 768, 512) for n in (1, 2, 16)] == [True, False, False]
    assert [takes(n, 2, 1024, 768) for n in (1, 2, 32)] == [True, False, False]
    assert [takes(n, 2, 1024, 960) for n in (1, 2, 4)] == [True, False, False]
    assert [takes(n, per, 2048, 2048) for n, per in ((1, 1), (1, 3), (8, 2))] == [False, False, False]


def test_only_weights_are_promised_to_stay_as_they_are_for_a_kernels_whole_life():
    """A kernel that starts while the one in front of it still runs must not promise that what that one writes is constant
    (``const T* __restrict__``): the compiler may then fetch it before the wait, or through a cache that is not coherent."""
    import re
    from pathlib import Path
    weights = {"sinks", "post_w", "layer_scale", "next_w", "weight", "w", "w2", "bias", "f_bias", "i_bias", "dt_bias", "a_log",
               "lower", "decay", "skip", "inv_freq", "table"}
    outputs = {"out", "y", "prep", "order", "tiles", "n_tiles", "pair_row", "tile_expert", "table", "rows", "gates", "token_ids",
               "positions", "req_kv_len"}
    found = 0
    for path in sorted(Path(ops.__file__).resolve().parent.glob("*.cu")):
        if path.name.endswith("probe.cu"):
            continue
        for promise in re.finditer(r"((?:const )?)([\w:]+)\* __restrict__ (\w+)", path.read_text()):
            const, kind, name = promise.groups()
            assert name in (weights if const else outputs), (path.name, promise.group(0))
            assert not (const and name == "table" and kind == "float2"), path.name       # the step's cosines and sines
            found += 1
    assert found > 30


def test_a_refused_prefill_still_joins_the_decode_attention_beside_it(monkeypatch):
    """In a mixed step the decode attention runs on a second stream; whatever ends the call, the current stream waits for it
    before the memory it writes can be given to anybody else."""
    import weakref
    from types import SimpleNamespace
    import pytest
    import torch
    from tokamak_b200.parts import attention
    log = []

    class Side:
        def join(self):
            log.append(("join", held() is not None))

    def decode(*args, side, **kw):
        nonlocal held
        scratch = torch.zeros(8)
        held = weakref.ref(scratch)
        log.append(("decode", isinstance(side, Side)))
        return scratch

    def refuse(*args, **kw):
        log.append(("prefill", held() is not None))
        raise ops.KernelError("refused")
    held = lambda: None
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    monkeypatch.setattr(attention, "_side_stream", lambda device: Side())
    for name, value in (("flush_chains", lambda: None), ("latent_kernel_takes", lambda *a: False), ("attention_decode", decode),
                        ("decode_kernel_takes", lambda *a: True), ("prefill_kernel_takes", lambda *a: True),
                        ("prefill_tc_kernel_takes", lambda *a: True), ("decode_uses_balanced", lambda *a: False),
                        ("attention_prefill_tc", refuse)):
        monkeypatch.setattr(ops, name, value)
    t = lambda *shape: torch.zeros(*shape, dtype=torch.bfloat16)
    step = SimpleNamespace(decode_items=torch.zeros(1), prefill_items=torch.zeros(3), prefill_tc=None, positions=None, tok_req=None,
                           req_slot=None, err=None, max_kv_len=256)
    view = SimpleNamespace(k=t(2, 1, 16, 64), v=t(2, 1, 16, 64), table=None)
    with pytest.raises(ops.KernelError, match="refused"):
        attention.paged_attention(t(4, 2, 64), t(4, 2, 64), view, step, scale=1.0, window=None)
    assert log == [("decode", True), ("prefill", True), ("join", True)]


def test_nothing_of_a_step_begins_before_the_step_is_described():
    """The decode attention reads positions and block tables before its wait on the kernel in front of it, so the kernels that
    write them must not let later ones begin: no early launch, and their writes out before they end."""
    from pathlib import Path
    text = (Path(ops.__file__).resolve().parent / "step_state.cu").read_text()
    kernels = text.split("__global__")[1:]
    assert len(kernels) == 2
    for kernel in kernels:
        body = kernel[:kernel.index("\n}\n")]
        assert "pdl_wait();" in body and "pdl_trigger" not in body
        assert body.rindex("__threadfence();") > max(body.rindex("rec[kRecComputed] ="), body.index("apply_updates("))
