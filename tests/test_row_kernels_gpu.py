"""Row kernels (norms, rotation + cache append) at the edges of their dispatch: few and many rows, short and long rows, and inputs whose base
is not 16-byte aligned."""

import pytest
import torch

from research_b200 import ops

pytestmark = pytest.mark.gpu


def _bf16(*shape, seed, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale).bfloat16()


@pytest.mark.parametrize("rows", [1, 148, 149, 700])
@pytest.mark.parametrize("d", [8, 248, 1024, 1032, 4096, 4104, 8192, 16384, 16392])
def test_rmsnorm_rows(rows, d):
    """Against 64 bits: two roundings to bf16 (at most 2^-8 of the value each) of a value whose scale is right to a few fp32 units."""
    x, w = _bf16(rows, d, seed=d, scale=3.0), _bf16(d, seed=rows)
    got = ops.rmsnorm(x.cuda(), w.cuda(), 1e-6).cpu().double()
    xd = x.double()
    want = xd * torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + 1e-6) * w.double()
    assert ((got - want).abs() <= want.abs() * 2.0 ** -6.9 + 1e-30).all()


@pytest.mark.parametrize("rows", [2, 148, 149, 600])
@pytest.mark.parametrize("d", [4, 130, 1020, 4096, 4100, 8192, 8196])
def test_layer_norm_rows(rows, d):
    g = torch.Generator().manual_seed(rows + d)
    y, x, w, b = (torch.randn(*s, generator=g) for s in ((rows, d), (rows, d), (d,), (d,)))
    want = x.double() + torch.nn.functional.layer_norm(y.double(), (d,), w.double(), b.double(), 1e-5)
    xg, xb = x.cuda(), torch.zeros(rows, d, dtype=torch.bfloat16, device="cuda")
    ops.layernorm_residual(y.cuda(), w.cuda(), b.cuda(), 1e-5, xg, xb)
    assert (xg.cpu().double() - want).abs().max() <= 3e-5 * want.abs().max()
    assert torch.equal(xb, xg.bfloat16())


@pytest.mark.parametrize("D,Hq,Hkv", [(64, 14, 2), (64, 1, 1), (128, 32, 8), (128, 3, 1), (64, 70, 5)])
@pytest.mark.parametrize("T", [1, 5, 67])
@pytest.mark.parametrize("norm", [False, True])
@pytest.mark.parametrize("odd", [False, True])
def test_rope_and_append(D, Hq, Hkv, T, norm, odd):
    """Bit for bit the reference without head norms (the same roundings); with them the row scale may differ in its last bit, which moves a
    rounding: one unit of bf16 (2^-7 of the value) in the normalised value, its product with the weight and each of the two rotated terms."""
    n = T * (Hq + 2 * Hkv) * D
    store = torch.zeros(n + 8, dtype=torch.bfloat16, device="cuda")
    qkv = store[1:n + 1] if odd else store[:n]            # contiguous; its base is 2 bytes off where odd
    qkv.copy_(_bf16(n, seed=T + D))
    qkv = qkv.view(T, -1)
    g = torch.Generator().manual_seed(T)
    pos = torch.randint(0, 300, (T,), generator=g, dtype=torch.int32)
    slots = torch.randperm(16 * 9, generator=g)[:T].int()
    slots[T // 2] = -1
    table = ops.rope_table(300, D, 1e4)
    qn, kn = (_bf16(D, seed=3), _bf16(D, seed=4)) if norm else (None, None)
    kc, vc = (torch.zeros(9, Hkv, 16, D, dtype=torch.bfloat16) for _ in range(2))
    kg, vg = kc.cuda(), vc.cuda()
    cuda = lambda t: None if t is None else t.cuda()       # noqa: E731
    q = ops.rope_kv_append(qkv, pos.cuda(), slots.cuda(), table.cuda(), kg, vg, Hq, Hkv, D, cuda(qn), cuda(kn))
    want = ops.rope_kv_append_reference(qkv.cpu(), pos, slots, table, kc, vc, Hq, Hkv, D, qn, kn)
    assert torch.equal(vg.cpu(), vc)
    for got, ref in ((q.cpu(), want), (kg.cpu(), kc)):
        if norm:
            assert (got.double() - ref.double()).abs().max() <= 4 * 2.0 ** -7 * ref.double().abs().max()
        else:
            assert torch.equal(got, ref)
