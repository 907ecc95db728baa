"""Products with few rows (csrc/skinny_sm100.cu) against 64-bit sums and against the tcgen05 kernel, over the forms both take."""

import pytest
import torch

from research_b200 import ops

gemm_mod = ops.gemm_mod


def _strided(rows, cols, pad, gen, scale=1.0):
    return (torch.randn(rows, cols + pad, device="cuda", generator=gen) * scale).bfloat16()[:, :cols]


def _reference(a, b, bias=None, residual=None, norm_eps=None, swiglu=False, bn=0, glu_limit=None, softcap=0.0, silu_cols=0, **_):
    """(result, bound on the sums' rounding), 64 bits; the bound is 2 K 2^-24 of the absolute sums, the worst order of fp32 additions."""
    x, w = a.double(), b.double()
    if norm_eps is not None:
        x = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + norm_eps)
    y, spread = x @ w.T, (x.abs() @ w.abs().T) * 2 * a.shape[1] * 2.0 ** -24
    if bias is not None:
        y = y + bias.double()
    if residual is not None:
        y = y + residual.double()
    if swiglu:
        v, s = y.view(len(y), -1, 2, bn // 2), spread.view(len(y), -1, 2, bn // 2)
        g, u = v[:, :, 0], v[:, :, 1]
        size = (g.abs() + 1) * (u.abs() + 2)
        # three roundings to bf16 on the way, and the sums' own error through both factors
        spread = (3 * 2.0 ** -9 * size + 2 * (s[:, :, 0] * (u.abs() + 2) + s[:, :, 1] * (g.abs() + 1))).reshape(len(y), -1)
        if glu_limit is not None:
            g, u = g.clamp(max=glu_limit), u.clamp(-glu_limit, glu_limit)
            y = g * torch.sigmoid(1.702 * g) * (u + 1)
        else:
            y = torch.nn.functional.silu(g) * u
        y = y.reshape(len(a), -1)
    if softcap > 0:
        y = softcap * torch.tanh(y / softcap)
    if silu_cols:
        y[:, :silu_cols] = torch.nn.functional.silu(y[:, :silu_cols])
    return y, spread


FORMS = {
    "plain": {},
    "f32": {"out_f32": True},
    "bias_residual": {"bias": True, "residual": True},
    "norm_bias": {"bias": True, "norm_eps": 1e-5},
    "softcap": {"out_f32": True, "softcap": 5.0},
    "silu_tail": {"silu_cols": 32, "tail": 8},
    "swiglu": {"swiglu": True, "bn": 64},
    "swiglu_norm": {"swiglu": True, "bn": 128, "norm_eps": 1e-6},
    "clamped": {"swiglu": True, "bn": 256, "glu_limit": 1.5},
}


@pytest.mark.parametrize("K", [64, 896])
def test_a_row_as_residual_is_left_to_the_general_path(K):
    """The general path takes the residual of a single row as a vector."""
    a, b = torch.zeros(1, K, dtype=torch.bfloat16), torch.zeros(128, K, dtype=torch.bfloat16)
    for residual, taken in ((torch.zeros(128, dtype=torch.bfloat16), False), (torch.zeros(1, 128, dtype=torch.bfloat16), True)):
        assert gemm_mod._few_rows_form(a, b, None, residual, 1, 128, K, 0, False, False, 0.0, 0, None) == taken


def test_sizes_at_which_few_row_kernels_pay():
    """The measured sides of every line of the rules: (M, N, K, gated unit, folded norm) -> kernel."""
    rows = lambda M, N, K, glu=False, norm=False: "skinny" if gemm_mod._skinny_pays(M, N, K, glu) else (
        "stream" if 9 <= M <= gemm_mod._stream_most_rows(N, K, glu, norm) else "one-CTA")
    for want, *sizes in (
            ("skinny", (1, 64, 64), (6, 151936, 896), (8, 128256, 4096), (16, 896, 4864), (16, 4096, 4096, False, True), (16, 2048, 128, True)),
            ("stream", (9, 28672, 4096), (9, 2048, 128), (12, 64, 64), (48, 32768, 256), (32, 2048, 512), (24, 16384, 512),
             (24, 9728, 2048), (40, 8192, 2048), (48, 37888, 1024), (64, 4096, 4096), (64, 896, 4864), (64, 28672, 4096, True), (64, 2048, 64, True)),
            ("one-CTA", (8, 151936, 896), (16, 2048, 128), (17, 2048, 256), (32, 64, 64), (64, 2048, 256), (64, 32768, 256), (48, 64, 512),
             (32, 16384, 512), (32, 9728, 896), (64, 9728, 896, False, True), (24, 9728, 2048, False, True), (32, 16384, 2048), (64, 28672, 4096), (64, 3072, 1024), (12, 151936, 896), (40, 128256, 4096, True))):
        for s in sizes:
            assert rows(*s) == want, (want, s, rows(*s))
    # gated units in blocks of 64, which the stream kernel does not take
    assert gemm_mod._skinny_pays(12, 28672, 4096, True, 64) and not gemm_mod._skinny_pays(12, 28672, 4096, True, 256)


@pytest.mark.gpu
@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("M", [1, 7, 8, 9, 16])
@pytest.mark.parametrize("N,K", [(8, 16), (72, 48), (136, 1040), (896, 4864), (4096, 64)])
def test_few_rows(form, M, N, K, monkeypatch):
    kw = dict(FORMS[form])
    if kw.get("swiglu"):
        N = -(-N // kw["bn"]) * kw["bn"]
    if kw.get("tail"):
        N += 64 - N % 32 + kw["tail"]
    gen = torch.Generator(device="cuda").manual_seed(M * 1000 + N + K)
    a, b = _strided(M, K, 16, gen), _strided(N, K, 32 if N < 1000 else 0, gen, K ** -0.5)
    if kw.pop("bias", False):
        kw["bias"] = torch.randn(N, device="cuda", generator=gen).bfloat16()
    if kw.pop("residual", False):
        kw["residual"] = _strided(M, N, 8, gen)
    tails = [torch.empty(M, kw["tail"] + 8, device="cuda")[:, :kw["tail"]] for _ in range(2)] if kw.get("tail") else [None, None]

    def run(tail):
        args = {k: v for k, v in kw.items() if k != "tail"}
        return ops.gemm(a, b, tail=tail, **args)

    monkeypatch.setattr(gemm_mod, "_skinny_pays", lambda *_: True)
    assert gemm_mod._skinny_takes(a, b, kw.get("bias"), kw.get("residual"), M, N, K, kw.get("bn", 0), kw.get("swiglu", False),
                                  kw.get("out_f32", False), kw.get("softcap", 0.0), kw.get("silu_cols", 0), tails[0])
    y, spread = _reference(a, b, **{k: v for k, v in kw.items() if k != "tail"})
    n = N - kw["tail"] if kw.get("tail") else y.shape[1]
    out = run(tails[0])
    half = 0.0 if kw.get("out_f32") else 2.0 ** -8
    # activations of softcap and silu: a few units in the last place of their fp32 value
    room = spread + half * y.abs() + 1e-6 * (1 + y.abs())
    assert ((out.double() - y[:, :n]).abs() <= room[:, :n]).all()
    if tails[0] is not None:
        assert ((tails[0].double() - y[:, n:]).abs() <= (spread + 1e-6)[:, n:]).all()
    monkeypatch.setattr(gemm_mod, "_skinny_pays", lambda *_: False)
    monkeypatch.setattr(gemm_mod, "_stream_most_rows", lambda *_: 0)
    other = run(tails[1])
    assert ((out.double() - other.double()).abs() <= 2 * room[:, :n]).all()


@pytest.mark.gpu
@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("M", [9, 16, 17, 32, 33, 64])
@pytest.mark.parametrize("N,K", [(8, 64), (136, 72), (896, 4864), (4096, 264)])
def test_up_to_64_rows(form, M, N, K, monkeypatch):
    """``rb_stream``: token counts around its steps of 16, K remainders and cuts, N below and above a tile."""
    kw = dict(FORMS[form])
    if kw.get("swiglu"):
        kw["bn"] = max(kw["bn"], 128)
        N = -(-N // kw["bn"]) * kw["bn"]
    if kw.get("tail"):
        N += 64 - N % 32 + kw["tail"]
    gen = torch.Generator(device="cuda").manual_seed(M * 1000 + N + K)
    a, b = _strided(M, K, 8, gen), _strided(N, K, 24, gen, K ** -0.5)
    if kw.pop("bias", False):
        kw["bias"] = torch.randn(N, device="cuda", generator=gen).bfloat16()
    if kw.pop("residual", False):
        kw["residual"] = _strided(M, N, 8, gen)
    tail = torch.empty(M, kw["tail"] + 8, device="cuda")[:, :kw["tail"]] if kw.get("tail") else None
    monkeypatch.setattr(gemm_mod, "_skinny_pays", lambda *_: False)
    monkeypatch.setattr(gemm_mod, "_stream_most_rows", lambda *_: 64)
    assert gemm_mod._stream_takes(a, b, kw.get("bias"), kw.get("residual"), M, N, K, kw.get("bn", 0), kw.get("swiglu", False),
                                  kw.get("out_f32", False), kw.get("softcap", 0.0), kw.get("silu_cols", 0), tail)
    out = ops.gemm(a, b, tail=tail, **{k: v for k, v in kw.items() if k != "tail"})
    y, spread = _reference(a, b, **{k: v for k, v in kw.items() if k != "tail"})
    n = N - kw["tail"] if kw.get("tail") else y.shape[1]
    room = spread + (0.0 if kw.get("out_f32") else 2.0 ** -8) * y.abs() + 1e-6 * (1 + y.abs())
    assert ((out.double() - y[:, :n]).abs() <= room[:, :n]).all()
    if tail is not None:
        assert ((tail.double() - y[:, n:]).abs() <= (spread + 1e-6)[:, n:]).all()
    ops.check_status(torch.device("cuda"))


@pytest.mark.gpu
@pytest.mark.parametrize("M", [4, 40])
def test_few_rows_under_capture_with_constant_weights(M):
    """First loads of the weights before the launch dependency is waited for: a chain in which every product reads the one before."""
    gen = torch.Generator(device="cuda").manual_seed(1)
    ws = [(torch.randn(512, 512, device="cuda", generator=gen) / 512 ** 0.5).bfloat16() for _ in range(6)]
    x = torch.randn(M, 512, device="cuda", generator=gen).bfloat16()
    bufs = [torch.empty(M, 512, device="cuda", dtype=torch.bfloat16) for _ in ws]

    def body():
        h = x
        for w, o in zip(ws, bufs):
            h = ops.gemm(h, w, out=o, constant_b=True)
        return h

    want = body().clone()
    ops.set_pdl(True)
    try:
        stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            body()
    finally:
        ops.set_pdl(False)
    for _ in range(20):
        for o in bufs:
            o.zero_()
        graph.replay()
        assert torch.equal(bufs[-1], want)


@pytest.mark.gpu
def test_waits_do_not_count_the_kernels_before():
    """Two products whose own bounded wait runs out (a flag that nothing sets) hold the stream for longer than the budget of one wait. The
    product behind them, which has started under them, still computes: its waits begin where theirs end."""
    from research_b200.ops._util import KernelStatusError

    gen = torch.Generator(device="cuda").manual_seed(3)
    a, slow_w = torch.randn(64, 128, device="cuda", generator=gen).bfloat16(), torch.randn(256, 128, device="cuda", generator=gen).bfloat16()
    x, w = torch.randn(32, 896, device="cuda", generator=gen).bfloat16(), torch.randn(896, 896, device="cuda", generator=gen).bfloat16()
    assert gemm_mod._stream_takes(x, w, None, None, 32, 896, 896, 0, False, False, 0.0, 0, None)
    want = ops.gemm(x, w)
    got, slow = torch.zeros_like(want), [torch.zeros(64, 256, device="cuda", dtype=torch.bfloat16) for _ in range(2)]
    flag = torch.tensor([0, 1], dtype=torch.int32, device="cuda")      # [0] the flag, [1] what it would have to reach
    torch.cuda.synchronize()
    ops.set_pdl(True)
    try:
        for o in slow:
            ops.gemm(a, slow_w, out=o, split_k=1, wait_flag=(flag.data_ptr(), flag.data_ptr() + 4))
        ops.gemm(x, w, out=got, constant_b=True)
    finally:
        ops.set_pdl(False)
    with pytest.raises(KernelStatusError):
        ops.check_status(torch.device("cuda"))
    assert torch.equal(got, want)
    ops.check_status(torch.device("cuda"))
