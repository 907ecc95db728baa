"""Products of 65 to 256 rows: gated units whose tiles take their gate and up rows as two boxes, and residuals added ahead of a cluster's reduction."""

import pytest
import torch

from research_b200 import ops

pytestmark = pytest.mark.gpu


def _bf16(*shape, seed, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda") * scale).bfloat16()


@pytest.mark.parametrize("M", [65, 128, 129, 256])
@pytest.mark.parametrize("N,K", [(256, 64), (1024, 200), (9472, 896), (18944, 128), (9728, 2048)])
@pytest.mark.parametrize("norm", [False, True])
@pytest.mark.parametrize("limit", [None, 7.0])
def test_gated_unit_tiles(M, N, K, norm, limit):
    """Tiles of 64, 128 and 256 columns of the same blocks give the same bits: the sums of a column do not depend on its tile."""
    x, w = _bf16(M, K, seed=M), _bf16(N, K, seed=N, scale=K ** -0.5)
    kw = dict(bn=256, swiglu=True, norm_eps=1e-6 if norm else None, glu_limit=limit)
    want = ops.gemm(x, w, max_ctas=147, **kw)          # a bounded grid keeps the wide tiles
    for constant in (False, True):
        assert torch.equal(ops.gemm(x, w, constant_b=constant, **kw), want)
    ops.check_status(torch.device("cuda"))


@pytest.mark.parametrize("M", [65, 100, 128])
@pytest.mark.parametrize("N,K", [(896, 896), (896, 4864), (904, 4864), (64, 2048), (2048, 4096)])
@pytest.mark.parametrize("shift", [0, 1])
def test_cluster_split_residual_and_bias(M, N, K, shift):
    """Rows of a residual or a bias that are not 16-byte aligned take single elements. Against 64 bits: a rounding of 2^-8 at most and sums of K
    products in fp32."""
    a, w = _bf16(M, K, seed=1), _bf16(N, K, seed=2, scale=K ** -0.5)
    res = _bf16(M, N + 8 + shift, seed=3)[:, shift:shift + N]
    bias = _bf16(N + 8, seed=4)[shift * 3:shift * 3 + N]
    split, bn = ops.gemm_mod._auto_split_k(M, N, K, False)
    assert split > 1
    got = ops.gemm(a, w, bias=bias, residual=res, constant_b=True).double()
    want = a.double() @ w.double().t() + bias.double() + res.double()
    assert ((got - want).abs() <= want.abs() * 2.0 ** -8 + 2e-5).all()
    ops.check_status(torch.device("cuda"))


def test_weights_ahead_of_the_launch_before():
    """A captured chain with programmatic launches: the activations that a product reads are those of the launch before it, every replay."""
    x = _bf16(128, 896, seed=1)
    ws = [_bf16(896, 896, seed=i + 2, scale=896 ** -0.5) for i in range(4)]
    wg = _bf16(9728, 896, seed=9, scale=896 ** -0.5)
    bufs = [torch.empty_like(x) for _ in ws]
    act = torch.empty(128, 4864, device="cuda", dtype=torch.bfloat16)

    def body():
        h = x
        for w, b in zip(ws, bufs):
            h = ops.gemm(h, w, out=b, residual=h, constant_b=True)
        ops.gemm(h, wg, out=act, bn=256, swiglu=True, norm_eps=1e-6, constant_b=True)

    ops.set_pdl(True)
    try:
        stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            body()
    finally:
        ops.set_pdl(False)
    for i in range(8):
        x.copy_(_bf16(128, 896, seed=100 + i))
        graph.replay()
        torch.cuda.synchronize()
        got = [b.clone() for b in (*bufs, act)]
        body()
        assert all(torch.equal(a, b) for a, b in zip(got, (*bufs, act)))
    ops.check_status(torch.device("cuda"))


@pytest.mark.parametrize("M", [1, 5, 8, 9, 16, 17, 31, 32, 33])
@pytest.mark.parametrize("N,K,form", [(19072, 896, {}), (20008, 904, dict(out_f32=True)), (38400, 896, dict(out_f32=True, softcap=30.0)),
                                      (19200, 1024, dict(bn=256, swiglu=True, norm_eps=1e-6)), (2048, 2048, {})])
def test_wide_outputs_of_few_rows(M, N, K, form):
    """Outputs of more than a tile an SM take rb_stream from one row on, others from nine. Against 64 bits, and no less exact than the one-CTA kernel."""
    x, w = _bf16(M, K, seed=M), _bf16(N, K, seed=N, scale=K ** -0.5)
    assert ops.gemm_mod._stream_first(M, N, K, bool(form.get("swiglu"))) == (M <= (64 if "swiglu" in form else 48 if N <= 37888 else 32) if N > 148 * 128 else 9 <= M <= 16)
    got, old = (ops.gemm(x, w, max_ctas=m, **form).double() for m in (0, 148))
    xd = x.double()
    if "norm_eps" in form:
        xd = xd * torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + 1e-6)
    want = xd @ w.double().t()
    if "softcap" in form:
        want = 30.0 * torch.tanh(want / 30.0)
    if "swiglu" in form:
        want = ops.gemm_mod.swiglu_interleaved_reference(want, 256, None)
    assert (got - want).norm() <= 1.05 * (old - want).norm()
    ops.check_status(torch.device("cuda"))
