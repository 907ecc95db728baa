"""Log-probabilities over a vocabulary: logits kept from the forward pass and logits multiplied out again give the same gradients."""

import pytest
import torch

from research_b200 import ops
from research_b200.ops import train as T
from research_b200.training.native_model import _FusedLogprob

pytestmark = pytest.mark.gpu


class _Sink:
    def __init__(self):
        self.seen = False

    def accumulate_into(self, view):
        before, self.seen = self.seen, True
        return before


@pytest.mark.parametrize("N,V,K", [(300, 1000, 128), (4096, 9600, 256), (4700, 4736, 320), (2049, 1001 * 8, 896)])
@pytest.mark.parametrize("entropy", [False, True])
def test_kept_logits_change_nothing(N, V, K, entropy):
    g = torch.Generator(device="cuda").manual_seed(N)
    h = torch.randn(N, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(V, K, device="cuda", generator=g) * K ** -0.5).bfloat16()
    t = torch.randint(0, V, (N,), device="cuda", generator=g, dtype=torch.int32)
    t[::7] = -1
    g_lp, g_ent = (torch.randn(N, device="cuda", generator=g) for _ in range(2))
    out = []
    for keep in (False, True):
        hh, gw = h.clone().requires_grad_(True), torch.full_like(w, float("nan"))
        lp, ent, _ = _FusedLogprob.apply(hh, w, gw, t, entropy, _Sink(), keep)
        torch.autograd.backward((lp, ent) if entropy else (lp,), (g_lp, g_ent) if entropy else (g_lp,))
        out.append((lp.detach(), ent.detach(), hh.grad, gw))
    for a, b in zip(*out):
        assert torch.equal(a, b)
    logits = h.double() @ w.double().t()
    p = logits.softmax(-1)
    lpd = logits.log_softmax(-1)
    valid = (t >= 0).double()[:, None]
    d = (g_lp.double()[:, None] * valid) * (torch.nn.functional.one_hot(t.long().clamp(min=0), V).double() - p)
    if entropy:
        d -= g_ent.double()[:, None] * p * (lpd - (p * lpd).sum(-1, keepdim=True))
    for got, want in ((out[1][2], d @ w.double()), (out[1][3], d.t() @ h.double())):
        assert (got.double() - want).norm() <= 6e-3 * want.norm()      # dlogits, result and one partial sum in bf16: 2^-8 at most each


def test_kept_only_where_a_backward_pass_may_come_and_memory_is_free():
    h = torch.zeros(64, 256, device="cuda", dtype=torch.bfloat16)
    assert not _FusedLogprob.keeps(h, 1000)
    h.requires_grad_(True)
    assert _FusedLogprob.keeps(h, 1000) and not _FusedLogprob.keeps(h, 1 << 40)
    with torch.no_grad():
        assert not _FusedLogprob.keeps(h, 1000)
    assert not _FusedLogprob.keeps(h.detach().cpu().requires_grad_(True), 1000)


@pytest.mark.parametrize("rows,V,pad", [(3, 8, 0), (5, 4096, 8), (2, 4104, 0), (4, 4097, 3), (3, 1003, 5)])
def test_gradient_of_logits_by_eights(rows, V, pad):
    """Rows whose length or stride is no multiple of eight take pairs; both against the same formula in 64 bits: one rounding to bf16 (2^-8 of the
    value at most), and fp32 exponentials and row sums good to about 1e-5 of their terms."""
    g = torch.Generator(device="cuda").manual_seed(V)
    x = torch.randn(rows, V + pad, device="cuda", generator=g)[:, :V] * 4
    t = torch.randint(0, V, (rows,), device="cuda", generator=g, dtype=torch.int32)
    t[0] = -1
    _, lse, ent = T.logprob_entropy_fwd(x, t, True)
    g_lp, g_ent = (torch.randn(rows, device="cuda", generator=g) for _ in range(2))
    out = torch.zeros(rows, V + pad, device="cuda", dtype=torch.bfloat16)
    T.logprob_entropy_bwd(x, t, lse, ent, g_lp, g_ent, out=out[:, :V])
    xd = x.double()
    p, lp = xd.softmax(-1), xd.log_softmax(-1)
    onehot = torch.nn.functional.one_hot(t.long().clamp(min=0), V).double()
    H = -(p * lp).sum(-1, keepdim=True)
    want = (g_lp.double() * (t >= 0))[:, None] * (onehot - p) - g_ent.double()[:, None] * p * (lp + H)
    terms = g_lp.double().abs()[:, None] * (onehot + p) + g_ent.double().abs()[:, None] * p * (lp.abs() + H)
    assert ((out[:, :V].double() - want).abs() <= want.abs() * 2.0 ** -8 + 2e-5 * terms).all()
    assert (out[:, V:] == 0).all()
    ops.check_status(torch.device("cuda"))
