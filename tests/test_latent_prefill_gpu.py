"""Prompt portions over a latent cache on tcgen05 (``latent_prefill.cuh``) against the formula in 64 bits: page sizes of every
loading shape, heads that do and do not divide the 128 rows of a block, portions that end inside a tile, a window that starts
inside a page, contexts before the portion, one to four stages of keys, and scores that grow along the keys, so that the
output is rescaled."""

from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu


def _i32(*values):
    return torch.tensor(values, dtype=torch.int32, device="cuda")


@pytest.mark.parametrize("T,ctx,H,rank,dr,page,window,sinks,dtype", [
    (1, 40, 3, 128, 0, 8, None, False, "float32"), (33, 0, 16, 512, 64, 16, None, True, "float32"),
    (70, 31, 5, 128, 64, 32, 1, False, "bfloat16"), (64, 0, 130, 128, 0, 16, None, True, "float32"),
    (130, 77, 16, 512, 0, 8, 45, True, "float32"), (200, 0, 1, 256, 64, 64, 100, False, "bfloat16"),
    (96, 260, 16, 384, 128, 96, None, True, "float32")])
@pytest.mark.parametrize("spread", [0.2, 6.0])
def test_portions_against_the_formula(T, ctx, H, rank, dr, page, window, sinks, dtype, spread):
    from tokamak_b200.csrc import ops
    g = torch.Generator().manual_seed(T + rank)
    D, L = rank + dr, ctx + T
    pages = -(-L // page)
    rows = torch.zeros(pages * page, D)
    rows[:L] = torch.randn(L, D, generator=g) * torch.linspace(0.2, 1.5, L)[:, None]
    rows = rows.bfloat16()
    perm = torch.randperm(pages + 1, generator=g)[:pages]
    cache = torch.full((pages + 1, 1, page, D), float("nan"), dtype=torch.bfloat16)
    cache[perm, 0] = rows.view(pages, page, D)
    table = torch.full((2, pages + 2), -1, dtype=torch.int32)
    table[1, :pages] = perm.int()
    if window is not None:
        table[1, :max(0, ctx - window + 1) // page] = -1          # pages that the window has passed are given back
    q = (spread * torch.randn(T, H, D, generator=g)).to(getattr(torch, dtype))
    start = 3                                                     # another request's tokens in front
    positions = torch.cat((torch.zeros(start), torch.arange(ctx, L))).int().cuda()
    step = SimpleNamespace(positions=positions, tok_req=_i32(*[0] * start, *[1] * T), req_q_start=_i32(0, start), req_q_len=_i32(start, T),
                           req_kv_len=_i32(start, L), req_slot=_i32(0, 1), err=_i32(0, 0, 0, 0))
    tiles = _i32(*[x for t in reversed(range(-(-T // 64))) for x in (1, t)])
    sink = torch.linspace(-1.0, 3.0, H) if sinks else None
    out = torch.full((start + T, H, rank), 7.0, dtype=torch.bfloat16, device="cuda")
    everything = torch.cat((torch.zeros(start, H, D, dtype=q.dtype), q)).cuda()
    scale = D ** -0.5
    for _ in range(2):
        ops.attention_latent(everything, out, cache.cuda(), rank, step, table.cuda(), scale=scale, window=window,
                             sinks=sink.cuda() if sinks else None, tiles=tiles)
    assert step.err.tolist()[0] == 0
    assert (out[:start] == 7.0).all()
    k = rows[:L].double()
    pos, key = torch.arange(ctx, L)[:, None], torch.arange(L)[None]
    seen = (key <= pos) & ((pos - key < window) if window else True)
    s = torch.einsum("thd,kd->htk", q.bfloat16().double(), k) * scale
    s = s.masked_fill(~seen, -torch.inf)
    if sinks:
        s = torch.cat((s, sink.double()[:, None, None].expand(H, T, 1)), -1)
    want = torch.einsum("htk,kd->thd", torch.softmax(s, -1)[..., :L], k[:, :rank])
    got = out[start:].double().cpu()
    # probabilities and results are rounded to 2^-9 of themselves: rows of several keys are 2e-3 off, 1e-2 is ample
    assert (got - want).norm() <= 1e-2 * want.norm()
    # and no more than the results' own rounding, to which float32 scores and sums of probabilities that keep 16 bits add 1e-5
    # of the value: the probabilities' rounding does not show
    assert (got - want).norm() <= 1.02 * (want.bfloat16().double() - want).norm() + 1e-4 * want.norm()


def _portion(rows, q, page, rank, sinks=None, dtype="float32"):
    """A whole prompt's attention over ``rows`` ``[keys, D]`` as a latent cache, ``q`` ``[keys, H, D]``."""
    from tokamak_b200.csrc import ops
    T, H, D = q.shape
    pages = -(-T // page)
    cache = torch.zeros(pages * page, D, dtype=torch.bfloat16)
    cache[:rows.shape[0]] = rows
    step = SimpleNamespace(positions=torch.arange(T, dtype=torch.int32, device="cuda"), tok_req=_i32(*[0] * T), req_q_start=_i32(0),
                           req_q_len=_i32(T), req_kv_len=_i32(T), req_slot=_i32(0), err=_i32(0, 0, 0, 0))
    out = torch.zeros(T, H, rank, dtype=torch.bfloat16, device="cuda")
    tiles = _i32(*[x for t in reversed(range(-(-T // 64))) for x in (0, t)])
    ops.attention_latent(q.to(getattr(torch, dtype)).cuda(), out, cache.view(pages, 1, page, D).cuda(), rank, step,
                         torch.arange(pages, dtype=torch.int32, device="cuda")[None].contiguous(), scale=D ** -0.5, sinks=sinks,
                         tiles=tiles)
    assert step.err.tolist()[0] == 0
    return out.cpu()


@pytest.mark.parametrize("low", [-torch.inf, torch.finfo(torch.float32).min, -2.5e38])
def test_a_sink_that_is_no_term_of_the_denominator(low):
    """As good as none: the same bits as without sinks, for heads beside one whose sink counts."""
    g = torch.Generator().manual_seed(5)
    rows, q = torch.randn(150, 192, generator=g).bfloat16(), torch.randn(150, 3, 192, generator=g)
    none = _portion(rows, q, 16, 128)
    got = _portion(rows, q, 16, 128, torch.tensor([low, 0.5, low], device="cuda"))
    assert torch.equal(got[:, [0, 2]], none[:, [0, 2]]) and (got[:, 1] != none[:, 1]).any()


@pytest.mark.parametrize("page", [8, 16, 32, 96])
@pytest.mark.parametrize("T,ctx,H,rank,dr,window", [(1, 0, 4, 128, 0, None), (70, 45, 16, 512, 64, 30), (20, 31, 3, 128, 64, 7)])
def test_rows_that_no_query_sees_may_hold_anything(T, ctx, H, rank, dr, window, page):
    """Behind the last position and in front of the window, in pages that are read: the same bits over NaN as over zeros."""
    from tokamak_b200.csrc import ops
    g = torch.Generator().manual_seed(page + T)
    D, L = rank + dr, ctx + T
    pages = -(-L // page)
    rows, q = torch.randn(L, D, generator=g).bfloat16(), torch.randn(T, H, D, generator=g).cuda()
    first = max(0, ctx - window + 1) if window else 0
    outs = []
    for behind in (0.0, float("nan")):
        cache = torch.full((pages * page, D), behind, dtype=torch.bfloat16)
        cache[first:L] = rows[first:]
        step = SimpleNamespace(positions=torch.arange(ctx, L, dtype=torch.int32, device="cuda"), tok_req=_i32(*[0] * T), req_q_start=_i32(0),
                               req_q_len=_i32(T), req_kv_len=_i32(L), req_slot=_i32(0), err=_i32(0, 0, 0, 0))
        out = torch.empty(T, H, rank, dtype=torch.bfloat16, device="cuda")
        ops.attention_latent(q, out, cache.view(pages, 1, page, D).cuda(), rank, step,
                             torch.arange(pages, dtype=torch.int32, device="cuda")[None].contiguous(), scale=D ** -0.5, window=window,
                             tiles=_i32(*[x for t in reversed(range(-(-T // 64))) for x in (0, t)]))
        assert step.err.tolist()[0] == 0
        outs.append(out.cpu())
    assert torch.isfinite(outs[0]).all() and torch.equal(*outs)


def test_a_page_outside_the_pool_is_reported():
    from tokamak_b200.csrc import ops
    cache = torch.zeros(2, 1, 16, 128, dtype=torch.bfloat16, device="cuda")
    step = SimpleNamespace(positions=torch.arange(20, dtype=torch.int32, device="cuda"), tok_req=_i32(*[0] * 20), req_q_start=_i32(0),
                           req_q_len=_i32(20), req_kv_len=_i32(20), req_slot=_i32(0), err=_i32(0, 0, 0, 0))
    out = torch.zeros(20, 2, 128, dtype=torch.bfloat16, device="cuda")
    ops.attention_latent(torch.zeros(20, 2, 128, device="cuda"), out, cache, 128, step, _i32(1, 9)[None], scale=1.0, tiles=_i32(0, 0))
    assert step.err.tolist()[0] == 2


def test_more_work_items_than_a_grid_has_planes():
    """Such a list goes to the kernel whose grid takes it: here the same tile over and over, which changes nothing."""
    from tokamak_b200.csrc import ops
    g = torch.Generator().manual_seed(2)
    rows, q = torch.randn(2, 128, generator=g).bfloat16(), torch.randn(2, 1, 128, generator=g)
    want = _portion(rows, q, 8, 128)
    cache = torch.zeros(8, 128, dtype=torch.bfloat16)
    cache[:2] = rows
    step = SimpleNamespace(positions=_i32(0, 1), tok_req=_i32(0, 0), req_q_start=_i32(0), req_q_len=_i32(2), req_kv_len=_i32(2),
                           req_slot=_i32(0), err=_i32(0, 0, 0, 0))
    out = torch.zeros(2, 1, 128, dtype=torch.bfloat16, device="cuda")
    tiles = torch.zeros(65536 * 2, dtype=torch.int32, device="cuda")
    ops.attention_latent(q.cuda(), out, cache.view(1, 1, 8, 128).cuda(), 128, step, _i32(0)[None], scale=128 ** -0.5, tiles=tiles)
    # two keys, probabilities rounded to bfloat16 in the other kernel: 2^-9 of each value, and the result's rounding
    torch.testing.assert_close(out.cpu().float(), want.float(), rtol=2.0 ** -7, atol=2.0 ** -7)


@pytest.mark.parametrize("offset", [0, 2])
def test_shares_of_a_single_token_are_added_up_into_rows_on_any_four_bytes(offset):
    from tokamak_b200.csrc import ops
    g = torch.Generator().manual_seed(9)
    L, H, D, page = 200, 3, 128, 16
    pages = -(-L // page)
    rows = torch.zeros(pages * page, D, dtype=torch.bfloat16)
    rows[:L] = torch.randn(L, D, generator=g).bfloat16()
    q = torch.randn(1, H, D, generator=g)
    step = SimpleNamespace(positions=_i32(L - 1), tok_req=_i32(0), req_q_start=_i32(0), req_q_len=_i32(1), req_kv_len=_i32(L), req_slot=_i32(0),
                           err=_i32(0, 0, 0, 0))
    memory = torch.zeros(H * D + 8, dtype=torch.bfloat16, device="cuda")
    out = memory[offset:offset + H * D].view(1, H, D)
    ops.attention_latent(q.cuda(), out, rows.view(pages, 1, page, D).cuda(), D, step, torch.arange(pages, dtype=torch.int32, device="cuda")[None],
                         scale=D ** -0.5, items=_i32(0), n_splits=3)
    k = rows[:L].double()
    want = torch.softmax(q[0].bfloat16().double() @ k.T * D ** -0.5, -1) @ k
    assert step.err.tolist()[0] == 0 and (memory[:offset] == 0).all() and (memory[offset + H * D:] == 0).all()
    torch.testing.assert_close(out[0].double().cpu(), want, rtol=1e-2, atol=5e-3)
