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


def _product(n, cols, parts, dt, g):
    """A product's result of ``cols`` columns as the kernels read it, and its value."""
    if not parts:
        x = torch.randn(n, cols, generator=g).to(dt)
        return x.to(DEV), x.double()
    x = torch.randn(parts, n, cols, generator=g)
    return x.to(DEV), x.double().sum(0)


# float32: a handful of roundings of values of size one and sums of up to 300 squares; bfloat16: the result's rounding
TOL = {"float32": dict(rtol=2e-5, atol=2e-5), "bfloat16": dict(rtol=2.0 ** -8, atol=2e-3)}


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("parts", [0, 1, 3])
@pytest.mark.parametrize("n,heads,dv", [(1, 1, 1), (8, 8, 256), (3, 2, 257), (150, 9, 40), (2, 3, 300)])
def test_output_stages_of_the_recurrences(n, heads, dv, parts, dtype):
    """Heads of up to 256 values are held by a warp, longer ones walked; a warp a block and four; partial sums and none."""
    from tokamak_b200.csrc import ops
    dt, g, cols = getattr(torch, dtype), torch.Generator().manual_seed(n + dv), heads * dv
    o, w = torch.randn(n, heads, dv, generator=g), torch.randn(cols, generator=g)
    proj, gate = _product(n, cols + 8, parts, dt, g)
    gate = gate[:, 8:].view(n, heads, dv)
    unit = lambda x: x * (x.square().mean(-1, keepdim=True) + 1e-5).rsqrt()
    got = ops.gla_out(o.to(DEV), proj, 8, w[:dv].to(DEV), 1e-5, dt, out_scale=0.5)
    want = unit(o.double()) * w[:dv].double() * torch.nn.functional.silu(gate) * 0.5
    torch.testing.assert_close(got.double().cpu(), want.view(n, cols), **TOL[dtype])
    last, gates = torch.randn(n, heads, 1, generator=g), torch.rand(n, heads, 3, generator=g)
    got = ops.mlstm_out(torch.cat((o, last), -1).to(DEV), gates.to(DEV), proj, 8, w.to(DEV), 1e-5, dt)
    h = o.double() / (torch.maximum(last.double().abs(), gates[..., 2:].double()) + 1e-6)
    want = unit(h) * w.double().view(heads, dv) * torch.sigmoid(gate)
    torch.testing.assert_close(got.double().cpu(), want.view(n, cols), **TOL[dtype])
    xbc, skip = torch.randn(n, cols + 4, generator=g), torch.randn(heads, generator=g)
    got = ops.ssd_out(o.to(DEV), xbc.to(DEV), proj, 8, skip.to(DEV), w.to(DEV), 1, 1e-5, dt)
    h = (o.double() + skip.double()[:, None] * xbc[:, :cols].double().view(n, heads, dv)) * torch.nn.functional.silu(gate)
    torch.testing.assert_close(got.double().cpu(), unit(h.view(n, cols)) * w.double(), **TOL[dtype])


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("width,outputs", [(64, 8), (2048, 16), (2048, 17), (2052, 8), (30, 4)])
def test_the_router_gives_a_token_the_same_bits_in_every_step(width, outputs, dtype):
    """Its rows are held by a warp each up to 2,048 wide and as many as a block has warps (16 in steps of few tokens, 8 otherwise), else
    walked in pieces; weights beside the formula."""
    from tokamak_b200.csrc import ops
    g = torch.Generator().manual_seed(width + outputs)
    h = torch.randn(200, width, generator=g).to(getattr(torch, dtype))
    router = torch.randn(outputs, width, generator=g) / width ** 0.5
    many = ops.moe_route(h.to(DEV), router.to(DEV), None, top=2)
    few = ops.moe_route(h[5:8].to(DEV).contiguous(), router.to(DEV), None, top=2)
    assert torch.equal(many.chosen[5:8], few.chosen) and torch.equal(many.weights[5:8], few.weights)
    scores = torch.sigmoid(h.double() @ router.double().T)
    want = scores.gather(1, many.chosen.long().cpu())
    torch.testing.assert_close(many.weights.double().cpu(), want, rtol=1e-5, atol=1e-5)
    torch.testing.assert_close(want.sum(1), scores.topk(2).values.sum(1), rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("parts", [0, 2])
@pytest.mark.parametrize("rank,cq", [(16, 0), (40, 1536), (512, 1537), (1600, 64)])
def test_cache_rows_and_query_latents_on_both_sides_of_the_registers(rank, cq, parts, dtype):
    """Six values a thread of up to 256 are held; the rest of a longer row is read again."""
    from tokamak_b200.csrc import ops
    dt, g, n = getattr(torch, dtype), torch.Generator().manual_seed(rank + cq), 3
    i32 = lambda *x: torch.tensor(x, dtype=torch.int32, device=DEV)
    proj, x = _product(n, rank + cq + 5, parts, dt, g)
    wk, wq = torch.randn(rank, generator=g), torch.randn(cq, generator=g)
    cache = torch.full((1, 1, 8, rank), 7.0, dtype=dt, device=DEV)
    err = i32(0, 0, 0, 0)
    _, latent = ops.latent_prepare(proj, cache, i32(2, 3, 4), i32(0, 0, 0), i32(0), i32(0)[None], err, kv_off=5, rank=rank, rot=0,
                                   kv_norm_w=wk.to(DEV), eps=1e-5, cq_off=5 + rank, cq_norm_w=wq.to(DEV) if cq else None)
    assert err.tolist()[0] == 0
    unit = lambda x: x * (x.square().mean(-1, keepdim=True) + 1e-5).rsqrt()
    torch.testing.assert_close(cache[0, 0, 2:5].double().cpu(), unit(x[:, 5:5 + rank]) * wk.double(), **TOL[dtype])
    assert (cache[0, 0, [0, 1, 5, 6, 7]] == 7).all()
    if cq:
        torch.testing.assert_close(latent.double().cpu(), unit(x[:, 5 + rank:]) * wq.double(), **TOL[dtype])


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("parts", [0, 2])
@pytest.mark.parametrize("channel", [False, True])
@pytest.mark.parametrize("heads,kv_heads,dk,dv,taps", [(1, 1, 4, 1, 2), (2, 1, 33, 70, 3), (4, 2, 128, 256, 4), (2, 2, 256, 40, 4)])
def test_inputs_of_the_delta_rule_for_single_tokens(heads, kv_heads, dk, dv, taps, channel, parts, dtype):
    """The kernel of such steps beside the one that takes a head a block, in values and in the moved tails, bit for bit."""
    from tokamak_b200.csrc import ops
    dt, g, n, slots = getattr(torch, dtype), torch.Generator().manual_seed(dk + dv), 3, 5
    hk, hv = kv_heads * dk, heads * dv
    proj, _ = _product(n, 2 * hk + hv + 2 * heads, parts, dt, g)
    floats, _ = ops.delta_record_floats(heads, kv_heads, dk, dv, taps)
    records = torch.randn(slots, floats, generator=g)
    i32 = lambda *x: torch.tensor(x, dtype=torch.int32, device=DEV)
    rand = lambda *s: torch.randn(*s, generator=g).to(DEV)
    w, a_log, dt_bias = rand(2 * hk + hv, taps), rand(heads), rand(heads * (dk if channel else 1))
    extra = dict(channel_a=_product(n, heads * dk, parts, dt, g)[0]) if channel else {}
    results = []
    for shape in (0, 2):
        rec, err = records.to(DEV), i32(0, 0, 0, 0)
        out = ops.delta_prepare(proj, w, a_log, dt_bias, rec, i32(0, 1, 2), i32(0, 1, 2), i32(1, 1, 1), i32(4, 0, 2), err, dtype=dt, q_off=0,
                                k_off=hk, v_off=2 * hk, b_off=2 * hk + hv, a_off=2 * hk + hv + heads, heads=heads, kv_heads=kv_heads,
                                key_dim=dk, value_dim=dv, unit_eps=1e-6, q_scale=dk ** -0.5, shape=shape, **extra)
        assert err.tolist()[0] == 0
        results.append((*out, rec))
    for a, b in zip(*results):
        assert torch.isfinite(a).all() and torch.equal(a, b)
    assert not torch.equal(results[0][-1][4].cpu(), records[4]) and torch.equal(results[0][-1][[1, 3]].cpu(), records[[1, 3]])


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("halves", [False, True])
@pytest.mark.parametrize("heads,rank,rot,cq", [(16, 32, 64, 0), (3, 40, 7, 0), (0, 64, 6, 200)])
def test_a_token_has_the_same_latent_rows_in_steps_of_every_size(heads, rank, rot, cq, halves, dtype):
    """The kernel that holds rows and the one for steps of many tokens; rotated pairs to the last bit, whose second member sums
    its products in another order in query rows than in cache rows."""
    from tokamak_b200.csrc import ops
    if halves and rot % 2:
        pytest.skip("halves are of one size")
    dt, g, n = getattr(torch, dtype), torch.Generator().manual_seed(rank + rot), 1300
    i32 = lambda *x: torch.tensor(x, dtype=torch.int32, device=DEV)
    pairs = rot // 2
    proj = torch.randn(n, rank + rot + heads * rot + cq, generator=g).to(dt)
    table, q_abs = torch.randn(n, pairs, 2, generator=g), torch.randn(max(heads, 1), n, rank, generator=g)
    wk, wq = torch.randn(rank, generator=g).to(DEV), torch.randn(cq, generator=g).to(DEV)

    def rows(k):
        pages = -(-k // 16)
        cache, err = torch.zeros(pages, 1, 16, rank + rot, dtype=dt, device=DEV), i32(0, 0, 0, 0)
        kw = dict(q_abs=q_abs[:, :k].contiguous().to(DEV), q_off=rank + rot, q_head_cols=rot) if heads else {}
        if cq:
            kw.update(cq_off=rank + rot, cq_norm_w=wq)
        q, c = ops.latent_prepare(proj[:k].to(DEV), cache, i32(*range(k)), i32(*[0] * k), i32(0), i32(*range(pages))[None], err, kv_off=0,
                                  rank=rank, rot=rot, kv_norm_w=wk, eps=1e-5, table=table[:k].to(DEV), halves=halves, **kw)
        assert err.tolist()[0] == 0
        return [x.cpu() for x in (cache.view(-1, rank + rot)[:k], q, c) if x is not None]

    many = rows(n)
    for a, b in zip(rows(5), many):
        assert torch.equal(a, b[:5])
    fma = lambda a, b, c: (a.double() * b.double() + c.double()).float()
    cos, sin = table[:, None, :, 0], table[:, None, :, 1]
    for got, x in ((many[0][:, None, rank:], proj[:, None, rank:rank + rot].float()),) + (
            ((many[1][:, :, rank:], proj[:, rank + rot:rank + rot + heads * rot].view(n, heads, rot).float()),) if heads else ()):
        first, second = ((slice(0, pairs), slice(pairs, rot)) if halves else (slice(0, 2 * pairs, 2), slice(1, 2 * pairs, 2)))
        u, w = x[..., first], x[..., second]
        c, s = cos.expand_as(u), sin.expand_as(u)
        query = x.shape[1] > 1
        assert torch.equal(got[..., first], fma(u, c, -(w * s)).to(got.dtype))
        assert torch.equal(got[..., second], (fma(u, s, w * c) if query and not halves else fma(w, c, u * s)).to(got.dtype))


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("hq,hkv,d,dv", [(16, 4, 128, 128), (2, 6, 40, 24), (3, 1, 200, 300)])
def test_a_token_has_the_same_normed_rows_in_steps_of_every_size(hq, hkv, d, dv, dtype):
    """Three blocks a token in steps of some hundred tokens, one in longer ones."""
    from tokamak_b200.csrc import ops
    dt, g, n, page = getattr(torch, dtype), torch.Generator().manual_seed(d), 700, 16
    nq, nk, nv = hq * d, hkv * d, hkv * dv
    proj, bias, norm = (torch.randn(*s, generator=g) for s in ((n, nq + nk + nv), (nq + nk + nv,), (nq + nk,)))
    proj = proj.to(dt)
    i32 = lambda *x: torch.tensor(x, dtype=torch.int32, device=DEV)
    cut = lambda t, a, b: t[a:b].to(DEV).contiguous()

    def rows(k):
        pages = -(-k // page)
        step = SimpleNamespace(positions=i32(*range(k)), tok_req=i32(*[0] * k), req_slot=i32(0), req_q_len=i32(k), req_kv_len=i32(k), err=i32(0, 0, 0, 0))
        kc, vc = (torch.full((pages, hkv, page, s), 7.0, dtype=dt, device=DEV) for s in (d, dv))
        q = torch.empty(k, hq, d, dtype=dt, device=DEV)
        ops.qkv_rownorm(proj[:k].to(DEV), q, kc, vc, step, i32(*range(pages))[None], q_off=0, k_off=nq, v_off=nq + nk, q_bias=cut(bias, 0, nq),
                        k_bias=cut(bias, nq, nq + nk), v_bias=cut(bias, nq + nk, None), q_norm=cut(norm, 0, nq), k_norm=cut(norm, nq, None), eps=1e-6)
        assert step.err.tolist()[0] == 0
        paged = lambda c, s: c.cpu().transpose(1, 2).reshape(pages * page, hkv * s)
        return q.cpu(), paged(kc, d), paged(vc, dv)

    many, some = rows(n), rows(100)        # both with 256 threads a row; a step of up to 64 tokens sums a row in another order
    for a, b in zip(some, many):
        assert torch.equal(a[:100], b[:100])
    assert (many[1][n:] == 0).all() and (many[2][n:] == 0).all()
    x = proj.double() + bias.double()
    want = x[:, :nq] * (x[:, :nq].square().mean(-1, keepdim=True) + 1e-6).rsqrt() * norm[:nq].double()
    torch.testing.assert_close(many[0].double().view(n, nq), want, **(dict(rtol=2e-5, atol=1e-6) if dtype == "float32" else dict(rtol=2.0 ** -8, atol=1e-6)))


@pytest.mark.parametrize("dv", [1, 64, 65, 128, 129, 256, 257])
def test_a_head_has_the_same_output_in_steps_of_every_size(dv):
    """Two, four, eight or no values of a head held by a lane; a warp a block and four."""
    from tokamak_b200.csrc import ops
    g, n, heads = torch.Generator().manual_seed(dv), 400, 4
    o, proj, w = (torch.randn(*s, generator=g).to(DEV) for s in ((n, heads, dv), (n, heads * dv), (heads * dv,)))
    gates, o1 = torch.rand(n, heads, 3, generator=g).to(DEV), torch.randn(n, heads, dv + 1, generator=g).to(DEV)
    for f in (lambda k: ops.gla_out(o[:k].contiguous(), proj[:k].contiguous(), 0, w[:dv].contiguous(), 1e-5, torch.float32),
              lambda k: ops.mlstm_out(o1[:k].contiguous(), gates[:k].contiguous(), proj[:k].contiguous(), 0, w, 1e-5, torch.float32)):
        assert torch.equal(f(3), f(n)[:3])
