"""Small kernels that hold a row in registers where it is short and walk it where it is long: either form against the same
arithmetic on the CPU, at widths on both sides of the line."""

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
