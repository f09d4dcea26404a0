"""Small kernels that hold a row in registers where it is short and walk it where it is long: either form against the same
arithmetic on the CPU, at widths on both sides of the line."""

from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


@pytest.mark.parametrize("parts", [0, 1, 2, 3])
@pytest.mark.parametrize("n,hidden,groups", [(1, 64, 4), (3, 2048, 8), (70, 2048, 8), (2, 4096, 2), (2, 4104, 3), (70, 4608, 8)])
def test_the_join_of_a_normed_branch_has_the_same_bits_at_every_size(n, hidden, groups, parts):
    """Eight elements whose squares sum to 32 have the root mean square two, so that the sum behind the norm can be told to
    the last bit: products with the weights, each rounded to float32, the last one into the sum with the stream before the
    rounding."""
    from tokamak_b200.csrc import ops
    g = torch.Generator().manual_seed(hidden + parts)
    eight = torch.tensor([5.0, 2.0, 1.0, 1.0, 1.0, 0.0, 0.0, 0.0])
    x = torch.cat([eight[torch.randperm(8, generator=g)] for _ in range(n * hidden // 8)]).view(n, hidden)
    x = torch.where(torch.rand(n, hidden, generator=g) < 0.5, -x, x)
    resid, post, scale, nxt = (torch.randn(*s, generator=g) for s in ((n, hidden), (hidden,), (hidden,), (hidden,)))
    branch = x
    if parts:
        branch = torch.randint(-4, 5, (parts, n, hidden), generator=g).float()
        branch[0] = x - branch[1:].sum(0)
    for weights in ((post, scale), (post, None), (None, scale), (None, None)):
        factors = [0.5] + [w for w in weights if w is not None]
        want = x
        for f in factors[:-1]:
            want = want * f
        want = (want.double() * factors[-1] + resid.double()).float()
        got, out = resid.to(DEV), torch.empty(n, hidden, device=DEV)
        ops.branch_norm_add(got, branch.to(DEV), *(None if w is None else w.to(DEV) for w in weights), 0.0, nxt.to(DEV), out, 1e-6,
                            branch_groups=groups, next_groups=groups)
        assert torch.equal(got.cpu(), want)
        v = want.double().view(n, groups, -1)
        normed = (v * (v.square().mean(-1, keepdim=True) + 1e-6).rsqrt()).view(n, hidden) * nxt.double()
        # two roundings of the result, and the sum's and the root's
        torch.testing.assert_close(out.double().cpu(), normed, rtol=8 * 2.0 ** -23, atol=1e-7)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("n,hq,hkv,d,dv", [(70, 2, 24, 128, 32), (3, 2, 72, 128, 16), (70, 24, 2, 128, 1100), (2, 1, 60, 4, 1000), (9, 4, 2, 64, 40)])
def test_rows_longer_than_the_registers(n, hq, hkv, d, dv, dtype):
    """Query, key and value rows on both sides of 8 values a thread (2,048 of a row, 8,192 in steps of up to 64 tokens), whichever of
    the three is the longest."""
    from tokamak_b200.csrc import ops
    dt = getattr(torch, dtype)
    g = torch.Generator().manual_seed(hkv * d + dv)
    nq, nk, nv = hq * d, hkv * d, hkv * dv
    proj = torch.randn(n, nq + nk + nv, generator=g).to(dt)
    bias, norm = torch.randn(nq + nk + nv, generator=g), torch.randn(nq + nk, generator=g)
    page = 16
    pages = -(-n // page)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    step = SimpleNamespace(positions=i32(list(range(n))), tok_req=i32([0] * n), req_slot=i32([0]), req_q_len=i32([n]), req_kv_len=i32([n]),
                           err=i32([0] * 4))
    k, v = (torch.full((pages, hkv, page, s), 7.0, dtype=dt, device=DEV) for s in (d, dv))
    q = torch.empty(n, hq, d, dtype=dt, device=DEV)
    cut = lambda t, a, b: t[a:b].to(DEV).contiguous()
    ops.qkv_rownorm(proj.to(DEV), q, k, v, step, i32([list(range(pages))]), q_off=0, k_off=nq, v_off=nq + nk, q_bias=cut(bias, 0, nq),
                    k_bias=cut(bias, nq, nq + nk), v_bias=cut(bias, nq + nk, None), q_norm=cut(norm, 0, nq), k_norm=cut(norm, nq, None), eps=1e-6)
    assert step.err.tolist()[0] == 0
    x = proj.double() + bias.double()
    normed = lambda t, w: t * (t.square().mean(-1, keepdim=True) + 1e-6).rsqrt() * w.double()
    # float32 sums of up to 9,216 squares, then a rounding to the type
    tol = dict(rtol=2e-5, atol=1e-6) if dtype == "float32" else dict(rtol=2.0 ** -8, atol=1e-6)
    torch.testing.assert_close(q.double().cpu().view(n, nq), normed(x[:, :nq], norm[:nq]), **tol)
    paged = lambda c, s: c.double().cpu().transpose(1, 2).reshape(pages * page, hkv * s)
    torch.testing.assert_close(paged(k, d)[:n], normed(x[:, nq:nq + nk], norm[nq:]), **tol)
    torch.testing.assert_close(paged(v, dv)[:n], x[:, nq + nk:], **tol)
    assert (paged(k, d)[n:] == 0).all() and (paged(v, dv)[n:] == 0).all()


@pytest.mark.parametrize("heads", [1, 65533, 65534])
def test_query_rows_of_as_many_heads_as_a_grid_has_planes(heads):
    from tokamak_b200.csrc import ops
    i32 = lambda *x: torch.tensor(x, dtype=torch.int32, device=DEV)
    q_abs = torch.randn(heads, 1, 4, device=DEV)
    cache = torch.zeros(1, 1, 8, 4, device=DEV)
    err = i32(0, 0, 0, 0)
    rows, _ = ops.latent_prepare(torch.ones(1, 4, device=DEV), cache, i32(3), i32(0), i32(0), i32(0)[None], err, kv_off=0, rank=4, rot=0,
                                 kv_norm_w=torch.ones(4, device=DEV), eps=0.0, q_abs=q_abs)
    assert err.tolist()[0] == 0 and torch.equal(rows[0], q_abs[:, 0])
    assert (cache[0, 0, 3] == 1).all() and (cache[0, 0, :3] == 0).all()
