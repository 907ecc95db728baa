"""Programmatic dependent launches: only kernels that wait for the launch before them are started with the attribute."""

import ctypes

import pytest
import torch

from research_b200 import _native, ops


def test_every_library_has_a_switch_of_its_own():
    """The static behind ``rb::pdl_enabled`` must not be a symbol that the loader can share between the libraries of a process."""
    built = [name for name in _native.LIBRARIES if _native.available(name)]
    if not built:
        pytest.skip("no library is built here")
    for name in built:
        with pytest.raises(ValueError):
            ctypes.c_bool.in_dll(_native.load(name), "_ZZN2rb11pdl_enabledEvE2on")


def test_tensor_memory_is_taken_before_dependents_start():
    """A kernel that releases its dependents first can find its columns taken by one that then waits for it. (Read from the sources: the hang
    itself would need the GPU.)"""
    found = 0
    for path in sorted([*_native.SRC_DIR.glob("*.cu"), *_native.SRC_DIR.glob("*.cuh")]):
        for body in path.read_text().split("__global__")[1:]:
            if "tmem_alloc(" in body and "pdl_launch_dependents()" in body:
                assert body.index("tmem_alloc(") < body.index("pdl_launch_dependents()"), (path.name, body[:80])
                found += 1
    assert found >= 8


@pytest.mark.gpu
@pytest.mark.parametrize("M", [512, 1024])
def test_two_cta_products_in_a_captured_chain(M):
    """Norm -> gated product -> product of the sizes that run on the two-CTA kernel, captured with the switch on as decode graphs
    are: every replay equals the eager result, also right after the norm's input and every buffer between have changed."""
    g = torch.Generator(device="cuda").manual_seed(M)
    d, f = 2048, 8192
    x = torch.randn(M, d, device="cuda", generator=g).bfloat16()
    norm = torch.randn(d, device="cuda", generator=g).bfloat16()
    wgu = (torch.randn(2 * f, d, device="cuda", generator=g) * d ** -0.5).bfloat16()
    wd = (torch.randn(5120, f, device="cuda", generator=g) * f ** -0.5).bfloat16()
    assert ops.gemm_mod._use_pair_kernel(M, 2 * f, d, False, False) and ops.gemm_mod._use_pair_kernel(M, 5120, f, False, False)
    h, act, out = (torch.empty(M, n, device="cuda", dtype=torch.bfloat16) for n in (d, f, 5120))

    def body():
        ops.rmsnorm(x, norm, 1e-6, out=h)
        ops.gemm(h, wgu, out=act, bn=256, swiglu=True, constant_b=True)
        ops.gemm(act, wd, out=out, constant_b=True)

    ops.set_pdl(True)
    try:
        stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            body()
    finally:
        ops.set_pdl(False)
    for i in range(12):
        x.normal_(generator=g)
        for t in (h, act, out):
            t.zero_()
        graph.replay()
        got = out.clone()
        body()
        assert torch.equal(got, out), i
