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
