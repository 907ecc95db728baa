"""Mixture-of-experts MLP for training as grouped tcgen05 GEMMs: forward, data gradients and weight gradients of ALL
experts of a layer run as six grouped launches over expert-sorted rows, with no host synchronisation.

The (token, slot) pairs are sorted by expert on the device; every expert's row range is padded with zero rows to a
multiple of 64, so the weight gradient ``dW_e = dY_e^T X_e`` is one grouped launch whose contraction runs over the
expert's row range (a 64-row k-block never straddles two experts). Rows keep the token order inside an expert, so the
result does not depend on scheduling.

Math of the per-expert loop in the reference's functional models
(rollouts/tools/functional_extractor/glm4_moe_functional.py:230-369: route, loop over experts, ``index_add_``);
``grouped_experts_reference`` below is that loop in fp32 and serves as the oracle and the CPU path.
"""

from __future__ import annotations

import ctypes

import torch

from .. import _native
from . import elementwise as _ew
from ._util import check_rc, status_tensor, stream_handle
from .gemm import EPI_STORE, RbGemmArgs, _lib as _gemm_lib, _lib2 as _gemm2_lib

_LIB = None
_I, _VP = ctypes.c_int, ctypes.c_void_p


def _lib():
    global _LIB
    if _LIB is None:
        lib = _native.load("rb_moe")
        lib.rb_moe_count.argtypes = [_VP, _I, _I, _VP, _VP]
        lib.rb_moe_train_plan.argtypes = [_VP, _I, _VP, ctypes.POINTER(_I), ctypes.POINTER(_VP), ctypes.POINTER(_VP), _I, _I, _I, _VP, _VP]
        lib.rb_moe_train_rows.argtypes = [_VP, _I, _I, _VP, _VP, _VP, _VP]
        lib.rb_moe_train_gather.argtypes = [_VP, _VP, _VP, _VP, _I, _I, _I, _VP, _VP]
        lib.rb_moe_train_combine.argtypes = [_VP, _VP, _VP, _I, _I, _I, _VP, _VP]
        lib.rb_moe_train_dot.argtypes = [_VP, _VP, _VP, _I, _I, _I, _VP, _VP]
        for f in ("rb_moe_count", "rb_moe_train_plan", "rb_moe_train_rows", "rb_moe_train_gather", "rb_moe_train_combine", "rb_moe_train_dot"):
            getattr(lib, f).restype = _I
        _LIB = lib
    return _LIB


MAX_EXPERTS = 256
FWD_GU, FWD_DN, DGRAD_DN, DGRAD_GU, WGRAD_DN, WGRAD_GU = range(6)


def _tile_width(n: int) -> int:
    return 256 if n >= 256 else 128 if n >= 128 else 64


def _pair_wgrad_pays(E: int, m: int, n: int, accumulate: bool) -> bool:
    """Weight gradients ``[m, n]`` of ``E`` experts on the two-CTA kernel's 256-row tiles (csrc/gemm2_sm100.cu) or on the one-CTA kernel's 128 rows.
    Microseconds, one-CTA / two-CTA. The two-CTA kernel reads less per product: E 128, 1536 x 2048 and 2048 x 768 508 / 385 at 64 rows an
    expert, E 256, 512 x 96 .75 of the time. Rows of a tile that the matrix does not have leave one CTA of the pair without an epilogue,
    which is what bounds short contractions: E 256, 128 x 1024 at 64 rows 30 / 46, adding 68 / 120; 384 x 1024 81 / 87, adding 211 / 240; 1024 x 32 19 / 23.
    Up to two waves of tiles that does not show (E 128, 64 x 256 .92; E 8, 64 x 64 .87). A single 128-column tile that is only written:
    E 256, 2048 x 128 at 192 rows 80 / 96, adding .91."""
    def up(x: int, step: int) -> int:
        return -(-x // step) * step

    columns = 128 if n <= 128 else 256
    pair = up(m, 256) * up(n, columns)
    if E * pair <= 148 * 256 * columns:
        return True
    return pair <= 1.25 * up(m, 128) * up(n, _tile_width(n)) and (accumulate or n != 128)


def _pair_tokens_pays(n: int, k: int, mn_major: bool) -> bool:
    """Products of the experts' rows with ``[n, k]`` weights on the two-CTA kernel, weights as its 256-row side, or on the one-CTA kernel's 128-row tiles.
    Microseconds (gate|up forward, down forward, their data gradients), one-CTA / two-CTA: 4096 tokens of 8 of 128 experts, 2048 x 768 238 / 207, 138 / 119,
    134 / 123, 240 / 203; 16 tokens 160 / 154, 88 / 86, 90 / 92, 146 / 145; 4096 of 2 of 8, 4096 x 3584 386 / 326, 210 / 169, 209 / 169, 406 / 331; 100 tokens
    108 / 111, 62 / 60, 60 / 61, 95 / 95; 64 of 2 of 8, 1024 x 1408, where the last tile of 1408 columns is half empty, 30 / 26, 28 / 19, 24 / 17, 38 / 28.
    Widths that would leave more of their tiles empty stay with the narrower ones."""
    return -(-n // 256) * 256 <= 1.15 * n and (k % 64 == 0 or not mn_major)


class GroupedPlan:
    """Row layout and tile tables of one MoE layer call, all on the device.

    ``idx`` ``[T, k]`` (int32) are the chosen experts. ``row_of[t * k + j]`` is the row of pair ``(t, j)`` in the
    expert-sorted matrices, ``src_of[row]`` its inverse (-1 for padding rows), ``offsets[e]`` the first row of expert
    ``e`` and ``offsets[E]`` the rows in use. ``cap`` is the fixed row capacity ``ceil64(T k) + 64 E`` the buffers
    are allocated with (the row count in use is only known on the device)."""

    def __init__(self, idx: torch.Tensor, E: int, d: int, F: int):
        assert idx.dtype == torch.int32 and idx.is_cuda and idx.is_contiguous() and E <= MAX_EXPERTS
        assert d % 64 == 0 and F % 32 == 0
        dev = idx.device
        self.T, self.k = idx.shape
        self.E, self.d, self.F, self.device = E, d, F, dev
        n = self.T * self.k
        self.n_pairs = n
        self.cap = -(-n // 64) * 64 + 64 * E
        lib, s = _lib(), stream_handle(dev)
        st = status_tensor(dev).data_ptr()
        self.counts = torch.zeros(E, dtype=torch.int32, device=dev)
        check_rc(lib.rb_moe_count(idx.data_ptr(), n, E, self.counts.data_ptr(), s), "rb_moe_count")
        # (mode, output columns per expert, tile width, rows of the stacked B per expert | output rows per expert)
        self.desc = [(0, 2 * F, _tile_width(2 * F), 2 * F), (0, d, _tile_width(d), d),
                     (1, F, _tile_width(F), d), (1, d, _tile_width(d), 2 * F),
                     (2, F, _tile_width(F), d), (2, d, _tile_width(d), 2 * F)]
        m_tiles = self.cap // 128 + E
        self.on_pair = {w for w in range(WGRAD_DN) if _pair_tokens_pays(self.desc[w][1], (d, F, d, 2 * F)[w], w >= DGRAD_DN)}
        for w in self.on_pair:
            self.desc[w] = (3, self.desc[w][1], 256, self.desc[w][3])
        # tables are written for the launches that read one
        used = [w for w in range(6) if w < WGRAD_DN or not _pair_wgrad_pays(E, self.desc[w][3], self.desc[w][1], False)]
        self.table_of = {which: table for table, which in enumerate(used)}
        written = [self.desc[which] for which in self.table_of]
        self.max_tiles = max((E * -(-bs // 128) if mode == 2 else self.cap // 256 + E if mode == 3 else m_tiles) * -(-n_total // bn)
                             for mode, n_total, bn, bs in written)
        tables = len(written)
        self.tiles = torch.empty(tables, self.max_tiles, 4, dtype=torch.int32, device=dev)
        self.ntiles = torch.zeros(tables, dtype=torch.int32, device=dev)
        self.offsets = torch.empty(E + 1, dtype=torch.int32, device=dev)
        flat = (_I * (4 * tables))(*[v for dsc in written for v in dsc])
        tptr = (_VP * tables)(*[self.tiles[i].data_ptr() for i in range(tables)])
        nptr = (_VP * tables)(*[self.ntiles.data_ptr() + 4 * i for i in range(tables)])
        check_rc(lib.rb_moe_train_plan(self.counts.data_ptr(), E, self.offsets.data_ptr(), flat, tptr, nptr, tables, self.max_tiles,
                                       self.cap, st, s), "rb_moe_train_plan")
        self.row_of = torch.empty(n, dtype=torch.int32, device=dev)
        self.src_of = torch.empty(self.cap, dtype=torch.int32, device=dev)
        check_rc(lib.rb_moe_train_rows(idx.data_ptr(), n, E, self.offsets.data_ptr(), self.row_of.data_ptr(),
                                       self.src_of.data_ptr(), s), "rb_moe_train_rows")

    # ---------------------------------------------------------------- token movement
    def gather(self, src: torch.Tensor, w: torch.Tensor | None = None) -> torch.Tensor:
        """``out[row] = (w[pair] if w else 1) * src[token of row]`` for the rows in use, zeros in the padding rows."""
        assert src.dtype == torch.bfloat16 and src.is_contiguous() and src.shape == (self.T, src.shape[1])
        cols = src.shape[1]
        out = torch.empty(self.cap, cols, dtype=torch.bfloat16, device=self.device)
        wp = None
        if w is not None:
            assert w.dtype == torch.float32 and w.is_contiguous() and w.numel() == self.n_pairs
            wp = w.data_ptr()
        check_rc(_lib().rb_moe_train_gather(src.data_ptr(), wp, self.src_of.data_ptr(), self.offsets.data_ptr() + 4 * self.E, self.cap,
                                            self.k, cols, out.data_ptr(), stream_handle(self.device)), "rb_moe_train_gather")
        return out

    def combine(self, y: torch.Tensor, w: torch.Tensor | None = None) -> torch.Tensor:
        """``out[t] = sum_j (w[t, j] if w else 1) * y[row_of[t, j]]``."""
        assert y.dtype == torch.bfloat16 and y.is_contiguous() and y.shape[0] == self.cap
        cols = y.shape[1]
        out = torch.empty(self.T, cols, dtype=torch.bfloat16, device=self.device)
        wp = None
        if w is not None:
            assert w.dtype == torch.float32 and w.is_contiguous() and w.numel() == self.n_pairs
            wp = w.data_ptr()
        check_rc(_lib().rb_moe_train_combine(y.data_ptr(), wp, self.row_of.data_ptr(), self.T, self.k, cols, out.data_ptr(),
                                             stream_handle(self.device)), "rb_moe_train_combine")
        return out

    def dot(self, g: torch.Tensor, y: torch.Tensor) -> torch.Tensor:
        """``dw[t, j] = <g[t], y[row_of[t, j]]>`` (fp32): the gradient of the combine weights."""
        assert g.is_contiguous() and y.is_contiguous() and g.shape[1] == y.shape[1]
        dw = torch.empty(self.T, self.k, dtype=torch.float32, device=self.device)
        check_rc(_lib().rb_moe_train_dot(g.data_ptr(), y.data_ptr(), self.row_of.data_ptr(), self.n_pairs, self.k, g.shape[1],
                                         dw.data_ptr(), stream_handle(self.device)), "rb_moe_train_dot")
        return dw

    # ---------------------------------------------------------------- grouped GEMMs
    def _launch(self, which: int, a, b, c, *, M, N, K, group_n, a_mn, b_mn, group_mode, group_b_rows=0, residual=None) -> None:
        args = RbGemmArgs()
        args.A[0], args.B[0], args.C = a.data_ptr(), b.data_ptr(), c.data_ptr()
        args.lda, args.ldb, args.ldc = a.stride(0), b.stride(0), c.stride(0)
        args.M, args.N, args.K = M, N, K
        args.a_parts = args.b_parts = 1
        args.a_mn_major, args.b_mn_major = int(a_mn), int(b_mn)
        args.bn = self.desc[which][2]
        args.epi_mode = EPI_STORE
        args.rank, args.world = 0, 1
        args.status = status_tensor(self.device).data_ptr()
        table = self.table_of[which]
        args.tile_table, args.num_tiles_ptr = self.tiles[table].data_ptr(), self.ntiles.data_ptr() + 4 * table
        args.group_n, args.max_tiles = group_n, self.max_tiles
        args.group_mode, args.group_b_rows = group_mode, group_b_rows
        if residual is not None:
            args.residual, args.ldr = residual.data_ptr(), residual.stride(0)
        check_rc(_gemm_lib().rb_gemm_bf16_ex(ctypes.byref(args), stream_handle(self.device)), "rb_gemm_bf16_ex(grouped training)")

    def _launch_pair(self, which: int, x, w, out, K: int, mn_major: bool) -> None:
        table = self.table_of[which]
        assert x.stride(1) == w.stride(1) == out.stride(1) == 1
        rc = _gemm2_lib().rb_gemm2_tokens(w.data_ptr(), x.data_ptr(), out.data_ptr(), self.E, out.shape[1], K, self.cap, int(mn_major), w.stride(0), x.stride(0),
                                          out.stride(0), self.tiles[table].data_ptr(), self.ntiles.data_ptr() + 4 * table, self.max_tiles,
                                          status_tensor(self.device).data_ptr(), stream_handle(self.device))
        check_rc(rc, "rb_gemm2_tokens")

    def forward(self, which: int, x: torch.Tensor, w: torch.Tensor) -> torch.Tensor:
        """``out[rows of e] = x[rows of e] @ w_e^T`` with ``w`` the experts' ``[n, K]`` matrices stacked along the rows."""
        n = self.desc[which][1]
        out = torch.empty(self.cap, n, dtype=torch.bfloat16, device=self.device)
        if which in self.on_pair:
            self._launch_pair(which, x, w, out, x.shape[1], False)
            return out
        self._launch(which, x, w, out, M=self.cap, N=w.shape[0], K=x.shape[1], group_n=n, a_mn=False, b_mn=False, group_mode=0)
        return out

    def dgrad(self, which: int, dy: torch.Tensor, w: torch.Tensor) -> torch.Tensor:
        """``out[rows of e] = dy[rows of e] @ w_e`` (``w_e`` is ``[K, n]``: the forward weight read MN-major)."""
        n = self.desc[which][1]
        kd = self.desc[which][3]
        assert dy.shape[1] == kd and w.shape == (self.E * kd, n)
        out = torch.empty(self.cap, n, dtype=torch.bfloat16, device=self.device)
        if which in self.on_pair:
            self._launch_pair(which, dy, w, out, kd, True)
            return out
        self._launch(which, dy, w, out, M=self.cap, N=n, K=kd, group_n=n, a_mn=False, b_mn=True, group_mode=1, group_b_rows=self.E * kd)
        return out

    def wgrad(self, which: int, dy: torch.Tensor, x: torch.Tensor, gw: torch.Tensor, accumulate: bool) -> None:
        """``gw_e (+)= dy[rows of e]^T @ x[rows of e]`` for every expert; ``gw`` is ``[E * m, n]``."""
        n, m = self.desc[which][1], self.desc[which][3]
        assert dy.shape == (self.cap, m) and x.shape == (self.cap, n) and gw.shape == (self.E * m, n)
        if not _pair_wgrad_pays(self.E, m, n, accumulate):
            self._launch(which, dy, x, gw, M=m, N=n, K=self.cap, group_n=n, a_mn=True, b_mn=True, group_mode=2,
                         residual=gw if accumulate else None)
            return
        assert gw.stride(1) == 1
        rc = _gemm2_lib().rb_gemm2_groups(dy.data_ptr(), x.data_ptr(), gw.data_ptr(), gw.data_ptr() if accumulate else None, self.E, m, n, self.cap,
                                          dy.stride(0), x.stride(0), gw.stride(0), gw.stride(0), self.offsets.data_ptr(),
                                          status_tensor(self.device).data_ptr(), stream_handle(self.device))
        check_rc(rc, "rb_gemm2_groups")


class GroupedExperts(torch.autograd.Function):
    """``out[t] = sum_j wt[t, j] * down_e(silu(gate_e x_t) * up_e x_t)``, ``e = idx[t, j]``.

    ``wgu`` ``[E * 2F, d]``: per expert the gate rows then the up rows; ``wd`` ``[E * d, F]``. ``ggu`` / ``gd`` are
    the gradient views the weight gradients are written into; ``sink.accumulate_into(view)`` says whether a view
    already holds gradients of this window (add) or is written for the first time (store)."""

    @staticmethod
    def forward(ctx, h, wt, wgu, ggu, wd, gd, plan: GroupedPlan, sink):
        xs = plan.gather(h)
        gu = plan.forward(FWD_GU, xs, wgu)
        act = _ew.swiglu(gu)
        y = plan.forward(FWD_DN, act, wd)
        wt = wt.contiguous()
        ctx.save_for_backward(xs, gu, y, wt, wgu, wd)
        ctx.plan, ctx.ggu, ctx.gd, ctx.sink = plan, ggu, gd, sink
        return plan.combine(y, wt)

    @staticmethod
    def backward(ctx, dout):
        xs, gu, y, wt, wgu, wd = ctx.saved_tensors
        plan: GroupedPlan = ctx.plan
        dout = dout.contiguous()
        dwt = plan.dot(dout, y) if ctx.needs_input_grad[1] else None
        dy = plan.gather(dout, wt)
        act = _ew.swiglu(gu)                                  # recomputed: cheaper than keeping [rows, F] alive
        plan.wgrad(WGRAD_DN, dy, act, ctx.gd, ctx.sink.accumulate_into(ctx.gd))
        dact = plan.dgrad(DGRAD_DN, dy, wd)
        del act, dy
        dgu = _ew.swiglu_backward(gu, dact)
        plan.wgrad(WGRAD_GU, dgu, xs, ctx.ggu, ctx.sink.accumulate_into(ctx.ggu))
        dh = None
        if ctx.needs_input_grad[0]:
            dh = plan.combine(plan.dgrad(DGRAD_GU, dgu, wgu))
        return dh, dwt, None, None, None, None, None, None


def grouped_experts_reference(h: torch.Tensor, idx: torch.Tensor, wt: torch.Tensor, wgu: torch.Tensor, wd: torch.Tensor) -> torch.Tensor:
    """The per-expert loop in fp32 (differentiable): the oracle of ``GroupedExperts`` and the path without a GPU."""
    T, d = h.shape
    E = wd.shape[0] // d
    F2 = wgu.shape[0] // E
    hf = h.float()
    out = torch.zeros(T, d, dtype=torch.float32, device=h.device)
    for e in range(E):
        tok, slot = (idx == e).nonzero(as_tuple=True)
        if tok.numel() == 0:
            continue
        gu = hf[tok] @ wgu[e * F2:(e + 1) * F2].float().t()
        g, u = gu[:, :F2 // 2], gu[:, F2 // 2:]
        y = (torch.nn.functional.silu(g) * u) @ wd[e * d:(e + 1) * d].float().t()
        out = out.index_add(0, tok, y * wt[tok, slot].float()[:, None])
    return out
