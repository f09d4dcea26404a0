"""Kernels whose work is split or laid out by the step's size: the same bits either way.  Segments of k in the true 32-bit
product; the recurrences' kernels for single tokens beside those for prompts, at sizes that end inside their tiles."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


@pytest.mark.parametrize("m,n,k", [(1, 65, 511), (17, 64, 512), (33, 130, 513), (64, 70, 1024), (65, 129, 2047), (5, 200, 2048),
                                   (130, 64, 3001), (16, 66, 4096)])
def test_segments_of_the_float32_product_give_the_same_bits(m, n, k):
    """A block for all segments of k and a block a segment, with every tile; beside float64: a sum of k products in segments
    rounds k times at most.  A row of C is the same whatever else is in the batch."""
    from tokamak_b200.csrc import ops
    for off in (0, 1):
        a = torch.randn(m * k + off, device=DEV)[off:].view(m, k)
        w = torch.randn(n * k + off, device=DEV)[off:].view(n, k)
        outs = [ops.gemm_f32(a, w, torch.full((m, n), float("nan"), device=DEV), tile=t) for t in (0, 1, 2, 3, 9, 10, 11)]
        assert all(torch.equal(o, outs[0]) for o in outs)
        bound = (a.double().abs() @ w.double().abs().T) * (k + 1) * 2.0 ** -24
        assert ((outs[0].double() - a.double() @ w.double().T).abs() <= bound).all()
        assert torch.equal(ops.gemm_f32(a[m // 2:m // 2 + 1].contiguous(), w)[0], outs[0][m // 2])


def _rows(*values):
    return torch.tensor(values, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("heads,dk,dv", [(1, 4, 1), (2, 3, 33), (3, 64, 30), (2, 100, 64), (2, 128, 257), (1, 200, 40), (2, 256, 96)])
def test_linear_scan_of_single_tokens(heads, dk, dv):
    """Requests in any slots; the state and the outputs of the prompt's kernel, and the formula in 64 bits."""
    from tokamak_b200.csrc import ops
    g = torch.Generator().manual_seed(dk + dv)
    n, slots = 5, 7
    dks, dvs = ops.gla_prepared_row(dk, dv)
    prep = torch.zeros(n * heads * (3 * dks + dvs))
    q, k, a = (torch.randn(heads, n, dk, generator=g) for _ in range(3))
    a, v = torch.sigmoid(a), torch.randn(heads, n, dv, generator=g)
    pieces = torch.zeros(heads, n, dks // 4, 3, 4)
    for i, x in enumerate((q, k, a)):
        pieces[:, :, :, i] = torch.nn.functional.pad(x, (0, dks - dk)).view(heads, n, dks // 4, 4)
    prep[:heads * n * 3 * dks] = pieces.flatten()
    prep[heads * n * 3 * dks:] = torch.nn.functional.pad(v, (0, dvs - dv)).flatten()
    state = torch.randn(slots, heads, dk, dv, generator=g)
    where = [4, 0, 6, 2, 5]
    err = torch.zeros(4, dtype=torch.int32, device=DEV)
    meta = (_rows(*range(n)), _rows(*[1] * n), _rows(*where), err)
    results = []
    for cols in (0, 8, 16, 32):
        s = state.to(DEV)
        results.append((ops.gla_scan(prep.to(DEV), s, *meta, cols=cols), s))
    assert err.tolist()[0] == 0
    for o, s in results[1:]:
        assert torch.equal(o, results[0][0]) and torch.equal(s, results[0][1])
    old = state[where].double()
    new = a.transpose(0, 1)[..., None].double() * old + k.transpose(0, 1)[..., None].double() * v.transpose(0, 1)[:, :, None].double()
    want = (new * q.transpose(0, 1)[..., None].double()).sum(2)
    torch.testing.assert_close(results[0][0].double().cpu(), want, rtol=1e-5, atol=1e-5 * dk ** 0.5)
    torch.testing.assert_close(results[0][1][where].double().cpu(), new, rtol=1e-5, atol=1e-5)
    untouched = [i for i in range(slots) if i not in where]
    assert torch.equal(results[0][1][untouched].cpu(), state[untouched])


@pytest.mark.parametrize("channel", [False, True])
@pytest.mark.parametrize("heads,kv_heads,dk,dv", [(1, 1, 4, 4), (2, 1, 32, 20), (4, 2, 100, 36), (2, 2, 128, 256), (2, 1, 256, 40)])
def test_delta_scan_of_single_tokens(heads, kv_heads, dk, dv, channel):
    """The kernel for single tokens beside the prompt's with either number of columns."""
    from tokamak_b200.csrc import ops
    g = torch.Generator().manual_seed(dk + dv)
    n, slots = 3, 4
    unit = lambda x: torch.nn.functional.normalize(x, dim=-1)
    q, k = (unit(torch.randn(n, kv_heads, dk, generator=g)) for _ in range(2))
    v, beta = torch.randn(n, heads, dv, generator=g), torch.rand(n, heads, generator=g)
    decay = torch.rand(*((n, heads, dk) if channel else (n, heads)), generator=g)
    records = torch.randn(slots, heads * dk * dv + 8, generator=g)       # a tail behind the state
    where = [3, 1, 0]
    err = torch.zeros(4, dtype=torch.int32, device=DEV)
    results = []
    for cols in (0, 16, 32):
        rec = records.to(DEV)
        o = ops.delta_scan(*(x.to(DEV) for x in (q, k, v, beta, decay)), rec, _rows(*range(n)), _rows(*[1] * n), _rows(*where), err,
                           cols=cols)
        results.append((o, rec))
    assert err.tolist()[0] == 0
    for o, rec in results[1:]:
        assert torch.equal(o, results[0][0]) and torch.equal(rec, results[0][1])
    S = records[where, :heads * dk * dv].view(n, heads, dk, dv).double()
    rep = lambda x: x.repeat_interleave(heads // kv_heads, 1).double()
    S = S * (decay.double()[..., None] if channel else decay.double()[..., None, None])
    u = beta.double()[..., None] * (v.double() - (S * rep(k)[..., None]).sum(2))
    S = S + rep(k)[..., None] * u[:, :, None]
    want = (S * rep(q)[..., None]).sum(2)
    torch.testing.assert_close(results[0][0].double().cpu(), want, rtol=1e-5, atol=1e-5 * dk ** 0.5)
    torch.testing.assert_close(results[0][1][where, :heads * dk * dv].view(n, heads, dk, dv).double().cpu(), S, rtol=1e-5, atol=2e-5)
