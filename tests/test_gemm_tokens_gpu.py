"""The product for a few hundred tokens (``gemm_tokens_tcgen05.cu``) against the same in 64 bits, at the edges of its
tiles: columns in steps of 16 and 32, one and two accumulators, columns staged in two parts, K splits of unequal length,
rows and k that end inside a tile, a second launch for the tiles that whole rounds leave over."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


def _run(tokens, n_out, k, **kw):
    from tokamak_b200.csrc import ops
    gen = torch.Generator().manual_seed(tokens + n_out + k)
    x = torch.randn(tokens, k, generator=gen).bfloat16()
    w = (torch.randn(n_out, k, generator=gen) / k ** 0.5).bfloat16()
    err = torch.zeros(4, dtype=torch.int32, device=DEV)
    got = ops.gemm_tokens(x.to(DEV), w.to(DEV), err, **kw)
    torch.cuda.synchronize()
    assert err.tolist()[0] == 0, err.tolist()
    return got.double().cpu(), x.double() @ w.double().T


# one rounding to bfloat16 (2^-9 of the value) and float32 sums: 1e-2 of the value and of sums of size one is ample
TOL = dict(rtol=1e-2, atol=1e-2)


@pytest.mark.parametrize("tokens,n_out,k,groups,splits", [
    (1, 256, 64, 1, 1), (16, 8, 8, 1, 1), (17, 264, 72, 1, 1), (65, 136, 200, 2, 1), (256, 512, 320, 1, 2), (257, 520, 576, 1, 3),
    (416, 256, 1024, 1, 4), (433, 384, 640, 1, 2), (512, 256, 448, 1, 4), (300, 1280, 520, 4, 2), (700, 640, 640, 2, 3)])
def test_given_groups_and_splits(tokens, n_out, k, groups, splits):
    got, want = _run(tokens, n_out, k, groups=groups, splits=splits)
    torch.testing.assert_close(got, want, **TOL)


# 80 tiles on 74 pairs of SMs leave six over, which run as a launch with more splits
@pytest.mark.parametrize("tokens,n_out,k", [(65, 1024, 1024), (208, 4104, 1000), (338, 20480, 2048), (1100, 512, 512)])
def test_own_plan(tokens, n_out, k):
    got, want = _run(tokens, n_out, k)
    torch.testing.assert_close(got, want, **TOL)


@pytest.mark.parametrize("activation", ["silu", "gelu_tanh"])
@pytest.mark.parametrize("tokens,inter,k,groups,splits", [(65, 64, 72, 1, 1), (200, 320, 640, 1, 3), (384, 192, 512, 1, 2),
                                                          (500, 128, 512, 1, 4), (338, 10240, 512, 0, 0)])
def test_gated_activation(tokens, inter, k, groups, splits, activation):
    got, sums = _run(tokens, 2 * inter, k, swiglu=True, activation=activation, groups=groups, splits=splits)
    sums = sums.view(tokens, inter // 64, 2, 64)
    g, u = sums[:, :, 0].reshape(tokens, -1), sums[:, :, 1].reshape(tokens, -1)
    act = torch.nn.functional.silu(g) if activation == "silu" else torch.nn.functional.gelu(g, approximate="tanh")
    torch.testing.assert_close(got, act * u, **TOL)


@pytest.mark.parametrize("tokens,n_out,k,splits", [(100, 384, 640, 2), (338, 264, 512, 4)])
def test_ungated_activation(tokens, n_out, k, splits):
    got, sums = _run(tokens, n_out, k, unary="relu2", groups=1, splits=splits)
    torch.testing.assert_close(got, torch.relu(sums) ** 2, rtol=1e-2, atol=2e-2)     # squares: twice the relative error


def test_what_the_rule_leaves_to_others():
    from tokamak_b200.csrc import ops
    x = torch.zeros(100, 128, dtype=torch.bfloat16, device=DEV)
    w = torch.zeros(256, 128, dtype=torch.bfloat16, device=DEV)
    assert ops.tokens_gemm_takes(x, w) and ops.tokens_gemm_takes(x.repeat(3, 1), w, fused=True)
    assert not ops.tokens_gemm_takes(x[:64], w)                                  # fewer tokens: the swapped product
    assert not ops.tokens_gemm_takes(x.repeat(3, 1), w)                          # more: the pairs of SMs or the library
    assert not ops.tokens_gemm_takes(x[:, 8:], w[:, 8:].contiguous())            # rows that do not follow one another
    assert not ops.tokens_gemm_takes(x, w[:, :120])
    flat = torch.zeros(100 * 128 + 1, dtype=torch.bfloat16, device=DEV)
    assert not ops.tokens_gemm_takes(flat[1:].view(100, 128), w)                 # not on a 16-byte boundary
    assert not ops.tokens_gemm_takes(x, w[:252]) and not ops.tokens_gemm_takes(x[:, :124].contiguous(), w[:, :124].contiguous())


@pytest.mark.parametrize("tokens,n_out,k", [(65, 1024, 1024), (140, 1024, 3072), (200, 4096, 4096), (338, 4104, 12288)])
def test_the_error_is_the_results_rounding(tokens, n_out, k):
    """Operands are exact and sums float32: what is left of the error, in the norm over all results, is the one rounding to
    bfloat16 (to which the sums add at most k roundings of 2^-24 a term, at random signs some 1e-6 of the result)."""
    got, want = _run(tokens, n_out, k)
    rounding = (want.bfloat16().double() - want).norm()
    assert (got - want).norm() <= 1.01 * rounding


@pytest.mark.parametrize("tokens,n_out,k,kw,launches", [(338, 20480, 2048, {}, 2), (338, 20480, 2048, dict(groups=1, splits=1), 1), (100, 256, 512, {}, 1)])
def test_launches_are_counted(tokens, n_out, k, kw, launches):
    """80 tiles on 74 pairs of SMs are two launches by the kernel's own plan."""
    from tokamak_b200.csrc import ops
    before = ops.LAUNCHES
    _run(tokens, n_out, k, **kw)
    assert ops.LAUNCHES - before == launches
