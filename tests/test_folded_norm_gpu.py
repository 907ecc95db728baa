"""Large products with a folded RMS norm: the rows' squares come from the product before, from a launch of their own, or not at all."""

import pytest
import torch

from research_b200 import ops

pytestmark = pytest.mark.gpu


def _bf16(*shape, seed, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda") * scale).bfloat16()


def _rel(got, want):
    return float((got.double() - want).norm() / want.norm())


@pytest.mark.parametrize("M", [512, 513, 2047, 2500])
@pytest.mark.parametrize("N,K,glu", [(9728, 896, True), (9720, 896, False), (4864, 264, False), (5120, 2048, True)])
def test_folded_norm_on_the_pair_kernel(M, N, K, glu):
    """Against 64 bits: a bf16 result is off by a rounding of at most 2^-8 (gated units: three), 2^-9.8 in the mean square; and by no more than the
    one-CTA kernel, which takes the squares from its operand tiles."""
    x, w, bias = _bf16(M, K, seed=1, scale=2.0), _bf16(N, K, seed=2, scale=K ** -0.5), _bf16(N, seed=3)
    assert ops.gemm_mod._use_pair_kernel(M, N, K, False, False)
    xd = x.double()
    want = (xd * torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + 1e-6)) @ w.double().t()
    kw = dict(norm_eps=1e-6, constant_b=True)
    if glu:
        kw |= dict(bn=256, swiglu=True)
        want = ops.gemm_mod.swiglu_interleaved_reference(want, 256, None)
    else:
        kw |= dict(bias=bias)
        want = want + bias.double()
    sq = ops.RowSquares(M, K, x.device)
    sq.measure(x)
    got, old = ops.gemm(x, w, squares=sq, **kw), ops.gemm(x, w, max_ctas=148, **kw)
    assert _rel(got, want) < (2.5 if glu else 1.2) * 2.0 ** -9.2
    assert _rel(got, want) < 1.02 * _rel(old, want)


@pytest.mark.parametrize("M,N,K", [(2816, 896, 4864), (2900, 904, 896), (512, 9728, 896), (600, 64, 256)])
def test_squares_left_by_a_product(M, N, K):
    """They add up to the squares of the rows as stored (fp32 sums of at most 9728 squares), and the product that takes them gives what it gives with
    squares measured from x; a product on another kernel marks them as unknown."""
    a, w, res = _bf16(M, K, seed=1), _bf16(N, K, seed=2, scale=K ** -0.5), _bf16(M, N, seed=3)
    sq = ops.RowSquares(M, N, a.device)
    sq.n = 99
    x = ops.gemm(a, w, residual=res, out=res, leave_squares=sq)
    if not ops.gemm_mod._use_pair_kernel(M, N, K, False, False):
        assert sq.n == 0
        return
    assert sq.n == -(-N // 256)
    got, want = sq.parts[:sq.n].double().sum(0), x.double().pow(2).sum(-1)
    assert ((got - want).abs() <= 2e-6 * want).all()
    w2 = _bf16(4096, N, seed=4, scale=N ** -0.5)
    one = ops.gemm(x, w2, norm_eps=1e-6, squares=sq)
    other = ops.RowSquares(M, N, a.device)
    other.measure(x)
    two = ops.gemm(x, w2, norm_eps=1e-6, squares=other)
    assert _rel(one, two.double()) < 1e-4      # single roundings of bf16 that a last bit of the row's scale moves
