"""tcgen05 flash attention (forward and backward) against fp32 PyTorch references."""

import math

import pytest
import torch

from research_b200 import ops
from research_b200.ops import flash

pytestmark = pytest.mark.gpu


def _rand(shape, device, seed, scale=1.0):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(shape, generator=g) * scale).to(torch.bfloat16).to(device)


def _cu(lens, device):
    return torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=device)


@pytest.mark.parametrize("D,Hq,Hkv", [(64, 14, 2), (128, 8, 2), (128, 4, 4)])
@pytest.mark.parametrize("causal,window", [(True, 0), (True, 100), (False, 0)])
def test_flash_varlen_forward(cuda_device, D, Hq, Hkv, causal, window):
    lens = [1, 127, 128, 129, 300, 517]
    T = sum(lens)
    # q, k, v as views of one fused projection output (row stride > H*D)
    qkv = _rand((T, (Hq + 2 * Hkv) * D), cuda_device, seed=1)
    q = qkv[:, : Hq * D].view(T, Hq, D)
    k = qkv[:, Hq * D : (Hq + Hkv) * D].view(T, Hkv, D)
    v = qkv[:, (Hq + Hkv) * D :].view(T, Hkv, D)
    cu = _cu(lens, cuda_device)
    got, lse = flash.flash_attn_varlen(q, k, v, cu, cu, max(lens), causal=causal, window=window, return_lse=True)
    want, lse_ref = flash.flash_attn_varlen_reference(q, k, v, cu, cu, causal=causal, window=window)
    diff = (got.float() - want.float()).abs()
    assert diff.max().item() < 0.02 and diff.mean().item() < 0.001, (diff.max().item(), diff.mean().item())
    assert torch.allclose(lse, lse_ref, atol=2e-3, rtol=1e-4), (lse - lse_ref).abs().max().item()


@pytest.mark.parametrize("D,Hq,Hkv", [(64, 14, 2), (128, 8, 2)])
def test_flash_cross_lengths(cuda_device, D, Hq, Hkv):
    """More keys than queries: the queries are the last positions (chunked prefill)."""
    q_lens, k_lens = [5, 64, 130, 1], [5, 200, 400, 77]
    q = _rand((sum(q_lens), Hq, D), cuda_device, seed=2)
    k = _rand((sum(k_lens), Hkv, D), cuda_device, seed=3)
    v = _rand((sum(k_lens), Hkv, D), cuda_device, seed=4)
    cu_q, cu_k = _cu(q_lens, cuda_device), _cu(k_lens, cuda_device)
    got = flash.flash_attn_varlen(q, k, v, cu_q, cu_k, max(q_lens))
    want, _ = flash.flash_attn_varlen_reference(q, k, v, cu_q, cu_k)
    diff = (got.float() - want.float()).abs()
    assert diff.max().item() < 0.02 and diff.mean().item() < 0.001, (diff.max().item(), diff.mean().item())


@pytest.mark.parametrize("D,Hq,Hkv", [(64, 14, 2), (128, 32, 8)])
@pytest.mark.parametrize("window", [0, 48])
def test_flash_paged_prefill(cuda_device, D, Hq, Hkv, window):
    new = [5, 64, 65, 130, 1, 200]
    prefix = [0, 16, 3, 100, 40, 0]
    lens = [n + p for n, p in zip(new, prefix)]
    B, bs = len(lens), 16
    nblk = [(l + bs - 1) // bs for l in lens]
    total = sum(nblk) + 3
    perm = torch.randperm(total, generator=torch.Generator().manual_seed(5))
    kc = _rand((total, Hkv, bs, D), cuda_device, seed=30)
    vc = _rand((total, Hkv, bs, D), cuda_device, seed=31)
    bt = torch.zeros(B, max(nblk) + 2, dtype=torch.int32)
    o = 0
    for b in range(B):
        bt[b, : nblk[b]] = perm[o : o + nblk[b]].to(torch.int32)
        o += nblk[b]
    bt = bt.to(cuda_device)
    cu = _cu(new, cuda_device)
    q = _rand((sum(new), Hq, D), cuda_device, seed=32)
    sl = torch.tensor(lens, dtype=torch.int32, device=cuda_device)
    got = flash.flash_paged_prefill(q, kc, vc, bt, cu, sl, max(new), window=window)
    want = ops.paged_prefill_reference(q, kc, vc, bt, cu, sl, window=window)
    diff = (got.float() - want.float()).abs()
    assert diff.max().item() < 0.02 and diff.mean().item() < 0.001, (diff.max().item(), diff.mean().item())


def test_flash_large_scores(cuda_device):
    """Scores that grow along the sequence exercise the lazy rescale of the O accumulator."""
    D, H, T = 128, 2, 1024
    q = _rand((T, H, D), cuda_device, seed=7, scale=3.0)
    k = _rand((T, H, D), cuda_device, seed=8, scale=3.0)
    k = (k.float() * torch.linspace(0.2, 3.0, T, device=cuda_device)[:, None, None]).to(torch.bfloat16)
    v = _rand((T, H, D), cuda_device, seed=9)
    cu = _cu([T], cuda_device)
    got, lse = flash.flash_attn_varlen(q, k, v, cu, cu, T, return_lse=True)
    want, lse_ref = flash.flash_attn_varlen_reference(q, k, v, cu, cu)
    diff = (got.float() - want.float()).abs()
    assert diff.max().item() < 0.03 and diff.mean().item() < 0.002, (diff.max().item(), diff.mean().item())
    assert torch.allclose(lse, lse_ref, atol=5e-3, rtol=1e-4)


def _grad_check(got, want, what, tol_max=0.06, tol_rel=0.02):
    diff = (got.float() - want.float()).abs()
    rel = diff.sum().item() / max(want.float().abs().sum().item(), 1e-9)
    assert diff.max().item() < tol_max and rel < tol_rel, (what, diff.max().item(), rel)


@pytest.mark.parametrize("D,Hq,Hkv", [(64, 14, 2), (128, 8, 2), (128, 4, 4)])
@pytest.mark.parametrize("causal,window", [(True, 0), (True, 100), (False, 0)])
def test_flash_varlen_backward(cuda_device, D, Hq, Hkv, causal, window):
    lens = [1, 63, 64, 129, 300, 517]
    T = sum(lens)
    qkv = _rand((T, (Hq + 2 * Hkv) * D), cuda_device, seed=11)
    q = qkv[:, : Hq * D].view(T, Hq, D)
    k = qkv[:, Hq * D : (Hq + Hkv) * D].view(T, Hkv, D)
    v = qkv[:, (Hq + Hkv) * D :].view(T, Hkv, D)
    dout = _rand((T, Hq, D), cuda_device, seed=12)
    cu = _cu(lens, cuda_device)
    out, lse = flash.flash_attn_varlen(q, k, v, cu, cu, max(lens), causal=causal, window=window, return_lse=True)
    dq, dk, dv = flash.flash_attn_varlen_backward(q, k, v, out, dout, lse, cu, cu, max(lens), max(lens), causal, window)
    qf, kf, vf = (t.detach().float().requires_grad_(True) for t in (q, k, v))
    o_ref, _ = flash.flash_attn_varlen_reference(qf, kf, vf, cu, cu, causal=causal, window=window)
    rq, rk, rv = torch.autograd.grad(o_ref, (qf, kf, vf), dout.float())
    _grad_check(dv, rv, "dv")
    _grad_check(dk, rk, "dk")
    _grad_check(dq, rq, "dq")


def test_flash_autograd_cross_lengths(cuda_device):
    D, Hq, Hkv = 128, 8, 2
    q_lens, k_lens = [5, 64, 130], [5, 200, 400]
    q = _rand((sum(q_lens), Hq, D), cuda_device, seed=13).requires_grad_(True)
    k = _rand((sum(k_lens), Hkv, D), cuda_device, seed=14).requires_grad_(True)
    v = _rand((sum(k_lens), Hkv, D), cuda_device, seed=15).requires_grad_(True)
    cu_q, cu_k = _cu(q_lens, cuda_device), _cu(k_lens, cuda_device)
    out = flash.flash_attention(q, k, v, cu_q, cu_k, max(q_lens), max(k_lens))
    w = _rand(out.shape, cuda_device, seed=16)
    (out.float() * w.float()).sum().backward()
    qf, kf, vf = (t.detach().float().requires_grad_(True) for t in (q, k, v))
    o_ref, _ = flash.flash_attn_varlen_reference(qf, kf, vf, cu_q, cu_k)
    rq, rk, rv = torch.autograd.grad(o_ref, (qf, kf, vf), w.float())
    _grad_check(v.grad, rv, "dv")
    _grad_check(k.grad, rk, "dk")
    _grad_check(q.grad, rq, "dq")


@pytest.mark.parametrize("D,Hq,Hkv", [(128, 4, 2), (64, 4, 1)])
@pytest.mark.parametrize("causal,window", [(True, 0), (True, 300), (False, 0)])
def test_flash_long_sequences_two_tile_kernel(cuda_device, D, Hq, Hkv, causal, window):
    """Lengths around multiples of 256 exercise the two-query-tile kernel: tile b missing, tile b with more key
    tiles than tile a, window starting inside tile a's range."""
    lens = [255, 256, 257, 1000, 1281]
    T = sum(lens)
    q, k, v = _rand((T, Hq, D), cuda_device, seed=21), _rand((T, Hkv, D), cuda_device, seed=22), _rand((T, Hkv, D), cuda_device, seed=23)
    cu = _cu(lens, cuda_device)
    got, lse = flash.flash_attn_varlen(q, k, v, cu, cu, max(lens), causal=causal, window=window, return_lse=True)
    want, lse_ref = flash.flash_attn_varlen_reference(q, k, v, cu, cu, causal=causal, window=window)
    diff = (got.float() - want.float()).abs()
    assert diff.max().item() < 0.02 and diff.mean().item() < 0.001, (diff.max().item(), diff.mean().item())
    assert torch.allclose(lse, lse_ref, atol=2e-3, rtol=1e-4), (lse - lse_ref).abs().max().item()


@pytest.mark.parametrize("D,Hq,Hkv", [(128, 8, 2), (64, 14, 2)])
def test_flash_backward_head_split(cuda_device, monkeypatch, D, Hq, Hkv):
    """dK/dV with one CTA per (key tile, query head) and a reduction over each group: same gradients as the
    per-kv-head form and as the fp32 reference; the automatic rule picks it only where the coarse grid has fewer CTAs than the GPU has SMs."""
    lens = [700, 129, 1]
    T = sum(lens)
    qkv = _rand((T, (Hq + 2 * Hkv) * D), cuda_device, seed=21)
    q = qkv[:, : Hq * D].view(T, Hq, D)
    k = qkv[:, Hq * D : (Hq + Hkv) * D].view(T, Hkv, D)
    v = qkv[:, (Hq + Hkv) * D :].view(T, Hkv, D)
    dout = _rand((T, Hq, D), cuda_device, seed=22)
    cu = _cu(lens, cuda_device)
    out, lse = flash.flash_attn_varlen(q, k, v, cu, cu, max(lens), causal=True, return_lse=True)
    monkeypatch.setattr(flash, "_HEAD_SPLIT", "0")
    base = flash.flash_attn_varlen_backward(q, k, v, out, dout, lse, cu, cu, max(lens), max(lens), True, 0)
    monkeypatch.setattr(flash, "_HEAD_SPLIT", "1")
    split = flash.flash_attn_varlen_backward(q, k, v, out, dout, lse, cu, cu, max(lens), max(lens), True, 0)
    qf, kf, vf = (t.detach().float().requires_grad_(True) for t in (q, k, v))
    o_ref, _ = flash.flash_attn_varlen_reference(qf, kf, vf, cu, cu, causal=True)
    rq, rk, rv = torch.autograd.grad(o_ref, (qf, kf, vf), dout.float())
    for got, want, what in zip(split, (rq, rk, rv), ("dq", "dk", "dv")):
        _grad_check(got, want, what + " (head split)")
    assert torch.equal(split[0], base[0])                       # dQ does not depend on the split
    for a, b in zip(split[1:], base[1:]):                       # fp32 sums over the group vs one accumulator: same to bf16 rounding
        assert (a.float() - b.float()).abs().max().item() < 0.02
    monkeypatch.setattr(flash, "_HEAD_SPLIT", "auto")
    assert flash.head_split_pays(1, 4096, 4096, 16, 2) and not flash.head_split_pays(1, 4096, 4096, 32, 8)
    assert not flash.head_split_pays(32, 512, 512, 14, 2) and not flash.head_split_pays(1, 4096, 4096, 8, 8)
    ops.check_status()


@pytest.mark.parametrize("paged", [False, True])
@pytest.mark.parametrize("D,H,Hkv,window", [(64, 14, 2, 0), (128, 8, 8, 0), (64, 6, 6, 200), (128, 4, 1, 129)])
def test_flash_forward_tile_edges_many_items_a_block(D, H, Hkv, window, paged):
    """More query tiles than the GPU has SMs, sequences around the tile sizes, empty ones and (paged) cached prefixes among them."""
    lens = [1, 127, 128, 129, 255, 256, 257, 0, 640, 1000, 383, 384, 385]
    prefix = [0, 5, 128, 0, 1, 130, 0, 7, 0, 16, 300, 0, 129] if paged else [0] * len(lens)
    g = torch.Generator(device="cuda").manual_seed(D + H + window)
    T, S = sum(lens), sum(lens) + sum(prefix)
    q = torch.randn(T, H, D, device="cuda", generator=g).bfloat16()
    k, v = (torch.randn(S, Hkv, D, device="cuda", generator=g).bfloat16() for _ in range(2))
    cu_q = torch.tensor([sum(lens[:i]) for i in range(len(lens) + 1)], dtype=torch.int32, device="cuda")
    kv = [a + b for a, b in zip(lens, prefix)]
    cu_k = torch.tensor([sum(kv[:i]) for i in range(len(kv) + 1)], dtype=torch.int32, device="cuda")
    lse = torch.empty(H, T, device="cuda")
    if paged:
        blocks = [-(-n // 16) for n in kv]
        order = torch.randperm(sum(blocks), generator=torch.Generator().manual_seed(1)).tolist()
        bt = torch.zeros(len(kv), max(blocks), dtype=torch.int32)
        kc, vc = (torch.zeros(sum(blocks), Hkv, 16, D, dtype=torch.bfloat16, device="cuda") for _ in range(2))
        at = 0
        for i, n in enumerate(kv):
            for j in range(blocks[i]):
                bt[i, j] = order[at]
                m = min(16, n - 16 * j)
                for cache, src in ((kc, k), (vc, v)):
                    cache[order[at], :, :m] = src[int(cu_k[i]) + 16 * j:int(cu_k[i]) + 16 * j + m].transpose(0, 1)
                at += 1
        out = ops.flash_paged_prefill(q, kc, vc, bt.cuda(), cu_q, torch.tensor(kv, dtype=torch.int32, device="cuda"), max(lens), window=window, lse=lse)
    else:
        out, lse = ops.flash_attn_varlen(q, k, v, cu_q, cu_k, max(lens), window=window, return_lse=True)
    ref, ref_lse = ops.flash_attn_varlen_reference(q.float(), k, v, cu_q, cu_k, window=window)
    size, _ = ops.flash_attn_varlen_reference(q.float(), k, v.abs(), cu_q, cu_k, window=window)
    # P and the output are rounded to bf16 (2^-8 each, relative); P's error meets every |v|
    assert ((out.float() - ref).abs() <= 2.0 ** -8 * size + 2.0 ** -8 * ref.abs() + 1e-6).all()
    assert ((lse - ref_lse).abs() <= 1e-4 * (1 + ref_lse.abs())).all()
    ops.check_status(torch.device("cuda"))


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("keys", [256, 384, 385, 512, 513, 640, 1411])
def test_flash_forward_second_tile_apart(keys, causal):
    """Query rows 128 to 255 are tile b, which starts late from four key tiles on. Alone they are tile a: the same key tiles in the same order, so the
    same bytes. Both against 64 bits: probabilities and the result in bf16, 2^-8 relative each, and the denominator is theirs in fp32."""
    D, H, Hkv, B = 64, 4, 2, 40
    q = _rand((B * 256, H, D), "cuda", seed=keys)
    k, v = (_rand((B * keys, Hkv, D), "cuda", seed=keys + i) for i in (1, 2))
    cu_q, cu_k, half = _cu([256] * B, "cuda"), _cu([keys] * B, "cuda"), _cu([128] * B, "cuda")
    both = flash.flash_attn_varlen(q, k, v, cu_q, cu_k, 256, causal=causal).view(B, 256, H, D)
    late = q.view(B, 256, H, D)[:, 128:].reshape(B * 128, H, D)
    assert torch.equal(both[:, 128:], flash.flash_attn_varlen(late, k, v, half, cu_k, 256, causal=causal).view(B, 128, H, D))
    kd, vd = (t.double().view(B, keys, Hkv, D).repeat_interleave(H // Hkv, 2) for t in (k, v))
    s = torch.einsum("bqhd,bkhd->bhqk", q.double().view(B, 256, H, D), kd) / math.sqrt(D)
    if causal:
        s = s.masked_fill(torch.arange(keys, device="cuda") > torch.arange(keys - 256, keys, device="cuda")[:, None], -math.inf)
    p = s.softmax(-1)
    want, terms = torch.einsum("bhqk,bkhd->bqhd", p, vd), torch.einsum("bhqk,bkhd->bqhd", p, vd.abs())
    assert ((both.double() - want).abs() <= 2.0 ** -8 * (want.abs() + terms) + 1e-4 * terms).all()
    ops.check_status(torch.device("cuda"))


@pytest.mark.parametrize("causal,window", [(True, 0), (True, 100), (True, 129), (False, 0)])
@pytest.mark.parametrize("D,H,Hkv", [(64, 4, 2), (128, 2, 2)])
def test_flash_backward_tile_edges(D, H, Hkv, causal, window):
    """Sequences around the 128-row tiles, an empty one, and one with more keys than queries, against 64 bits."""
    q_lens = [1, 127, 128, 129, 0, 255, 256, 257, 60, 383]
    k_lens = [1, 127, 128, 129, 0, 255, 256, 257, 200, 383]
    g = torch.Generator(device="cuda").manual_seed(D + window)
    q, do = (torch.randn(sum(q_lens), H, D, device="cuda", generator=g).bfloat16() for _ in range(2))
    k, v = (torch.randn(sum(k_lens), Hkv, D, device="cuda", generator=g).bfloat16() for _ in range(2))
    cu_q, cu_k = _cu(q_lens, "cuda"), _cu(k_lens, "cuda")
    out, lse = flash.flash_attn_varlen(q, k, v, cu_q, cu_k, max(q_lens), causal=causal, window=window, return_lse=True)
    got = flash.flash_attn_varlen_backward(q, k, v, out, do, lse, cu_q, cu_k, max(q_lens), max(k_lens), causal=causal, window=window)
    u = 2.0 ** -8        # a rounding to bf16
    at_q = at_k = 0
    for nq, nk in zip(q_lens, k_lens):
        want = [torch.zeros(n, h, D, device="cuda", dtype=torch.float64) for n, h in ((nq, H), (nk, Hkv), (nk, Hkv))]
        room = [torch.zeros_like(w) for w in want]
        for h in range(H):
            kv = h // (H // Hkv)
            qh, oh, dh = (t[at_q:at_q + nq, h].double() for t in (q, out, do))
            kh, vh = k[at_k:at_k + nk, kv].double(), v[at_k:at_k + nk, kv].double()
            i, j = torch.arange(nq, device="cuda")[:, None] + nk - nq, torch.arange(nk, device="cuda")[None]
            dead = (j > i) if causal else torch.zeros(nq, nk, dtype=torch.bool, device="cuda")
            dead = dead | (j <= i - window) if window else dead
            p = (qh @ kh.T * D ** -0.5).masked_fill(dead, -math.inf).softmax(-1)
            exact_o = p @ vh
            ds = p * (dh @ vh.T - (dh * exact_o).sum(-1, keepdim=True)) * D ** -0.5
            # dS is rounded; its delta is taken from the rounded output
            slack = u * ds.abs() + p * D ** -0.5 * (u * (dh.abs() * (p @ vh.abs())).sum(-1, keepdim=True) + 1e-5)
            want[0][:, h] = ds @ kh
            want[1][:, kv] += ds.T @ qh
            want[2][:, kv] += p.T @ dh
            room[0][:, h] = slack @ kh.abs()
            room[1][:, kv] += slack.T @ qh.abs()
            room[2][:, kv] += u * p.T @ dh.abs()
        for x, w, m, (lo, n) in zip(got, want, room, ((at_q, nq), (at_k, nk), (at_k, nk))):
            assert ((x[lo:lo + n].double() - w).abs() <= m + u * w.abs() + 1e-5).all()
        at_q, at_k = at_q + nq, at_k + nk
    ops.check_status(torch.device("cuda"))


def test_flash_in_a_thread_without_context(cuda_device):
    """A thread whose first CUDA call is the kernel's (autograd's may be one: its memory can all come from the cache)."""
    import threading

    q, k, v, do = (torch.randn(183, h, 128, device=cuda_device).bfloat16() for h in (4, 2, 2, 4))
    cu = torch.tensor([0, 183], dtype=torch.int32, device=cuda_device)
    out, lse = flash.flash_attn_varlen(q, k, v, cu, cu, 183, return_lse=True)
    want = [t.cpu() for t in flash.flash_attn_varlen_backward(q, k, v, out, do, lse, cu, cu, 183, 183)]      # (its memory goes back to the cache)
    got = []

    def work():
        try:
            got.append(flash.flash_attn_varlen_backward(q, k, v, out, do, lse, cu, cu, 183, 183))
        except RuntimeError as e:
            got.append(e)

    t = threading.Thread(target=work)
    t.start()
    t.join()
    assert isinstance(got[0], tuple), got[0]
    assert all(torch.equal(a.cpu(), b) for a, b in zip(got[0], want))
    ops.check_status(cuda_device)
