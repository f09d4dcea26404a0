"""Runs of equal layers launched from one native call against the same layers launched part by part: the same kernels with the
same arguments, so the same bits, in steps of every kind (prompt portions, single tokens, both; few and many tokens; 32-bit)."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _config(layers, dim, tied=False):
    return {"architectures": ["Qwen3ForCausalLM"], "num_hidden_layers": layers, "hidden_size": 256, "num_attention_heads": 4,
            "num_key_value_heads": 2, "head_dim": dim, "intermediate_size": 384, "vocab_size": 512, "rope_theta": 10000.0,
            "rms_norm_eps": 1e-6, "tie_word_embeddings": tied, "max_position_embeddings": 4096}


def _core(raw, dtype, page=16):
    from tokamak_b200.config import architecture_of
    from tokamak_b200.engine.core import EngineCore
    from tokamak_b200.models.decoder import DecoderModel
    from tokamak_b200.weights.random_init import random_tensors
    arch = architecture_of(raw)
    expected = DecoderModel.expected_tensors(arch.build_spec(arch.parse(raw)))
    w = random_tensors(expected, 3, 0.06, 0.1, getattr(torch, dtype), device="cuda")
    for name, req in expected.items():
        if name in w and req.role == "vector":
            w[name] = w[name].float()
    return EngineCore("<random>", dtype=dtype, tensors=w, raw_config=raw, max_seq_len=2048, page_size=page, pool_tokens=8192,
                      max_slots=6, max_step_tokens=1024)


def _steps(core, sizes, native):
    """Logits of prompt steps, of a step that mixes a portion with single tokens, and of single tokens alone; and how many kernels
    were launched."""
    from tokamak_b200.csrc import ops
    from tokamak_b200.engine.step import StepEntry
    model = core.step.model
    runs, model._runs = model._runs, model._runs if native else {}
    gen = torch.Generator().manual_seed(7)
    before, outs = ops.LAUNCHES, []
    try:
        prompts = [torch.randint(0, 512, (n,), generator=gen).tolist() for n in sizes]
        outs.append(core.step.run([StepEntry(i, p, [len(p) - 1]) for i, p in enumerate(prompts)]))
        if len(sizes) > 1:
            outs.append(core.step.run([StepEntry(0, prompts[0], [0, len(prompts[0]) - 1])]
                                      + [StepEntry(i, [i], [0]) for i in range(1, len(sizes))]))
            outs.append(core.step.run([StepEntry(i, [i + 9], [0]) for i in range(len(sizes))]))
        for i in range(len(sizes)):
            core.step.free(i)
    finally:
        model._runs = runs
    return outs, ops.LAUNCHES - before


@pytest.mark.parametrize("dtype,dim,layers,sizes", [
    ("bfloat16", 128, 6, [40]), ("bfloat16", 128, 6, [30, 17, 9]), ("bfloat16", 128, 2, [64]), ("bfloat16", 128, 6, [65]),
    ("bfloat16", 128, 9, [90, 60, 50]), ("bfloat16", 64, 5, [30, 5]), ("bfloat16", 64, 5, [120, 70]), ("float32", 128, 5, [30, 40]),
    ("float32", 64, 3, [200]), ("float32", 32, 2, [3, 1])])
def test_the_same_bits_as_part_by_part(dtype, dim, layers, sizes):
    core = _core(_config(layers, dim), dtype)
    assert core.step.model._runs == {0: layers}
    parts, launched = _steps(core, sizes, False)
    native, launched_native = _steps(core, sizes, True)
    assert launched == launched_native > 0
    for a, b in zip(parts, native):
        assert torch.isfinite(a).all() and torch.equal(a, b)


@pytest.mark.parametrize("sizes", [[300, 200], [512], [700, 100]])
def test_steps_in_which_another_product_may_be_taken(sizes):
    """Beyond a few hundred tokens the native call takes this library's product where the parts take the library's: two
    correctly rounded results of each product, so logits as far apart as bfloat16 activations make them."""
    core = _core(_config(4, 128), "bfloat16")
    parts, _ = _steps(core, sizes, False)
    native, _ = _steps(core, sizes, True)
    for a, b in zip(parts, native):
        assert (a - b).norm() <= 0.03 * a.norm()


def test_runs_end_where_layers_differ():
    from tokamak_b200.models.decoder import LayerCall, StreamInput
    from tokamak_b200.parts.dense_run import find_runs
    model = _core(_config(5, 128), "bfloat16").step.model
    calls = list(model.spec.schedule)
    assert find_runs(model.blocks, calls) == {0: 5}
    joined = calls[:3] + [LayerCall(calls[3].block, calls[3].cache, StreamInput(embedding=True))] + calls[4:]
    assert find_runs(model.blocks, joined) == {0: 3}
    sub = type("Sub", (type(model.blocks[calls[2].block]),), {})
    blocks = dict(model.blocks)
    blocks[calls[2].block].__class__ = sub
    assert find_runs(blocks, calls) == {0: 2, 3: 2}


def _off_by_one_element(t):
    out = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)[1:].view(t.shape)
    return out.copy_(t)


@pytest.mark.parametrize("change", ["misaligned", "transposed", "last layer only", "next norm"])
def test_what_only_the_library_takes_runs_part_by_part(change):
    """Matrices that this library's products cannot address, and a norm behind the run whose weight is of another type: the
    step runs as it does without the native call, and nothing is done twice."""
    core = _core(_config(6, 128), "bfloat16")
    model = core.step.model
    blocks = [model.blocks[c.block] for c in model.spec.schedule]
    if change == "next norm":
        norm = model.final_norm

        class Halved:
            spec, weight = norm.spec, norm.weight.bfloat16()
            add_norm = staticmethod(norm.add_norm)

        model.final_norm = Halved
    for block in (blocks[-1:] if change == "last layer only" else blocks if change != "next norm" else []):
        for part, name in ((block.mixer, "w_o"), (block.feed_forward, "w_down")):
            w = getattr(part, name)
            setattr(part, name, w.t().contiguous().t() if change == "transposed" else _off_by_one_element(w))
    parts, launched = _steps(core, [100], False)
    native, launched_native = _steps(core, [100], True)
    assert launched == launched_native
    for a, b in zip(parts, native):
        assert torch.isfinite(a).all() and torch.equal(a, b)


@pytest.mark.parametrize("dtype,tokens", [("bfloat16", 512), ("bfloat16", 64), ("float32", 300)])
def test_no_more_memory_than_part_by_part(dtype, tokens):
    """The most that is allocated during a step; rows of all parts at once would be two thirds more."""
    core = _core(_config(4, 128), dtype)
    most = {}
    for native in (False, True):
        for _ in range(2):                        # workspaces that stay are there from the first step on
            torch.cuda.synchronize()
            torch.cuda.reset_peak_memory_stats()
            before = torch.cuda.memory_allocated()
            _steps(core, [tokens], native)
            most[native] = torch.cuda.max_memory_allocated() - before
    assert most[True] <= most[False] + 65536, most          # rounding of the pieces, and the record of a step of few tokens


def _varied(core, change, monkeypatch):
    """The model of ``core`` with one thing about its layers changed, for the native run and the parts alike; the layers that the
    native run then has."""
    import dataclasses
    from types import SimpleNamespace
    from tokamak_b200.csrc import ops
    from tokamak_b200.parts.dense_run import find_runs
    model = core.step.model
    calls = list(model.spec.schedule)
    blocks = [model.blocks[c.block] for c in calls]
    for block in blocks:
        m, f = block.mixer, block.feed_forward
        if change == "window":
            m.spec = dataclasses.replace(m.spec, window=20)
        elif change == "gelu":
            f.spec = dataclasses.replace(f.spec, activation="gelu_tanh")
        elif change == "no q/k norm":
            m.spec = dataclasses.replace(m.spec, qk_norm_eps=None)
            m.q_norm_w = m.k_norm_w = None
        elif change == "half a head turned":
            whole, d = m.position.rotary_table, m.spec.head_dim
            m.position = SimpleNamespace(rotary_table=lambda step, w=whole, d=d: (w(step)[0][:, :d // 4].contiguous(), d // 2))
    if change == "balanced":
        monkeypatch.setattr(ops, "DECODE_ATTENTION", "balanced")
    elif change == "last norm":
        model.final_norm.__class__ = type("Sub", (type(model.final_norm),), {})
    elif change == "first layer":
        blocks[0].__class__ = type("Sub", (type(blocks[0]),), {})
    model._runs = find_runs(model.blocks, calls)
    return sum(model._runs.values())


@pytest.mark.parametrize("sizes", [[30, 17, 9], [90, 60, 50]])
@pytest.mark.parametrize("change,dim,page", [("balanced", 128, 16), ("window", 128, 16), ("gelu", 128, 16), ("no q/k norm", 128, 16), ("pages of 64", 128, 64),
                                             ("last norm", 128, 16), ("first layer", 128, 16), ("half a head turned", 64, 16),
                                             ("window", 64, 32)])
def test_the_same_bits_in_other_layers(change, dim, page, sizes, monkeypatch):
    """What differs between designs, and where a run begins behind other layers (with an owed norm in steps of few tokens) or
    ends in front of a norm that is not known."""
    from tokamak_b200.csrc import ops
    core = _core(_config(5, dim), "bfloat16", page)
    layers = _varied(core, change, monkeypatch)
    assert layers == (4 if change == "first layer" else 5)
    parts, launched = _steps(core, sizes, False)
    seen, launch = [], ops.dense_layers
    monkeypatch.setattr(ops, "dense_layers", lambda rows, want, step: (seen.append((step.mode, step.dec_kind, len(rows))), launch(rows, want, step)))
    native, launched_native = _steps(core, sizes, True)
    assert launched == launched_native > 0
    for a, b in zip(parts, native):
        assert torch.isfinite(a).all() and torch.equal(a, b)
    # prompts, a portion beside single tokens, single tokens; heads of 64 have no native form in steps of few tokens
    few = [sum(sizes) <= 64, sizes[0] + len(sizes) - 1 <= 64, True]
    kind = 2 if change == "balanced" else 1
    want = []
    for is_few, decodes in zip(few, (False, True, True)):
        if is_few and dim != 128:
            continue
        run = layers - (1 if is_few and change == "last norm" else 0)
        want += [(0 if is_few else 1, kind if decodes else 0, min(4, run - i)) for i in range(0, run, 4)]
    assert seen == want


def test_a_run_behind_other_layers_is_entered_with_an_owed_norm(monkeypatch):
    from tokamak_b200.models import decoder
    from tokamak_b200.parts.base import OwedNorm
    core = _core(_config(4, 128), "bfloat16")
    assert _varied(core, "first layer", monkeypatch) == 3
    entered, run = [], decoder.run_layers
    monkeypatch.setattr(decoder, "run_layers", lambda calls, resid, pending, *rest: (entered.append(type(pending)), run(calls, resid, pending, *rest))[1])
    _steps(core, [40], True)
    _steps(core, [100], True)
    assert entered == [OwedNorm, torch.Tensor]
