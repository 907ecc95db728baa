"""The vocabulary product whose epilogue is the gradient of the log-probabilities (csrc/gemm2_sm100.cu)."""

import pytest
import torch

from research_b200 import ops
from research_b200.ops import train as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("entropy", [False, True])
@pytest.mark.parametrize("M,N,K,scale", [(512, 9600, 256, 1.0), (513, 20008, 264, 6.0), (600, 19000, 896, 1.0), (2048, 4736, 320, 2.0)])
def test_vocabulary_dlogits_equal_the_two_kernels(M, N, K, scale, entropy):
    """Bit for bit what the product and the gradient kernel give; edges of the 256 x 256 tiles, ignored targets, strided rows."""
    g = torch.Generator(device="cuda").manual_seed(M + N)
    h = torch.randn(M, K + 16, device="cuda", generator=g).bfloat16()[:, :K]
    w = (torch.randn(N, K, device="cuda", generator=g) * scale * K ** -0.5).bfloat16()
    t = torch.randint(0, N, (M,), device="cuda", generator=g, dtype=torch.int32)
    t[::5] = -1
    t[1], t[2] = N - 1, 0
    g_lp, g_ent = (torch.randn(M, device="cuda", generator=g) for _ in range(2))
    assert ops.gemm_mod.vocabulary_takes(h, w)
    logits = ops.gemm(h, w, out_f32=True)
    _, lse, ent = T.logprob_entropy_fwd(logits, t, entropy)
    args = (t, lse, ent, g_lp, g_ent if entropy else None)
    got = ops.gemm_mod.vocabulary_dlogits(h, w, *args)
    want = T.logprob_entropy_bwd(logits, *args)
    assert torch.equal(got, want)
    ops.check_status(torch.device("cuda"))


def test_vocabulary_dlogits_leave_small_products_alone():
    h, w = (torch.zeros(n, 256, device="cuda", dtype=torch.bfloat16) for n in (511, 9600))
    assert not ops.gemm_mod.vocabulary_takes(h, w) and not ops.gemm_mod.vocabulary_takes(h.float(), w)


@pytest.mark.parametrize("V", [1, 300, 512, 513, 1537, 2047, 4095, 4096, 4097, 9000])
def test_row_sums_at_the_ends_of_their_rounds(V):
    """Row lengths around the rounds of loads, with masked and equal values; infinities and NaN come out as sums taken one by one give them."""
    g = torch.Generator(device="cuda").manual_seed(V)
    x = torch.randn(12, V, device="cuda", generator=g) * 20
    x[0] = 3.0
    x[1, 1:] = -float("inf")
    x[2, : V // 2] = -float("inf")
    x[3] = -float("inf")
    x[4, -1], x[5, 0] = float("nan"), float("inf")
    t = torch.randint(0, V, (12,), device="cuda", generator=g, dtype=torch.int32)
    logprob, lse, _ = T.logprob_entropy_fwd(x, t, False)
    want = torch.logsumexp(x.double(), 1)
    ok = torch.ones(12, dtype=torch.bool, device="cuda")
    ok[3:6] = False
    # at most V roundings of a running sum of positive terms, and exponentials good to a few units in the last place
    room = (V + 16) * 2.0 ** -24 + 2.0 ** -22 * (1 + want.abs())
    assert ((lse.double() - want).abs() <= room)[ok].all()
    assert ((logprob.double() - (x.double().gather(1, t.long()[:, None])[:, 0] - want)).abs() <= 2 * room)[ok & (logprob > -1e30)].all()
    # an infinite value makes the sum undefined, and so does a NaN behind a finite value of the same thread (512 columns before)
    assert lse[4].isnan() or V <= 512
    assert lse[3].isnan() or lse[3] == -float("inf")
    assert lse[5].isnan()
