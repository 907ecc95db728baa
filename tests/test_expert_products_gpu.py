"""Products of the experts' rows with the weights as the 256-row side of the two-CTA kernel's tile, against 64 bits and the one-CTA kernel."""

import pytest
import torch

from research_b200 import ops
from research_b200.ops import moe_train as M

pytestmark = pytest.mark.gpu


def _choices(rows: list[int]) -> torch.Tensor:
    """Every token to one expert, so that expert ``e`` gets ``rows[e]`` rows, in a mixed order."""
    idx = torch.cat([torch.full((n,), e, dtype=torch.int32) for e, n in enumerate(rows)])
    return idx[torch.randperm(len(idx), generator=torch.Generator().manual_seed(len(idx)))][:, None].contiguous().cuda()


@pytest.mark.parametrize("rows", [[1], [64, 0, 65, 256], [257, 1, 512, 513, 3, 300, 129, 320], [1, 2, 3, 1000], [31] * 70, [2100, 5]])
@pytest.mark.parametrize("d,F", [(256, 128), (512, 192), (1024, 1408), (2048, 768), (320, 96)])
def test_rows_of_experts(rows, d, F, monkeypatch):
    E, T = len(rows), sum(rows)
    idx = _choices(rows)
    g = torch.Generator(device="cuda").manual_seed(T)
    x, dy = (torch.randn(T, n, device="cuda", generator=g).bfloat16() for n in (d, 2 * F))
    act, dout = (torch.randn(T, n, device="cuda", generator=g).bfloat16() for n in (F, d))
    wgu = (torch.randn(E * 2 * F, d, device="cuda", generator=g) * d ** -0.5).bfloat16()
    wd = (torch.randn(E * d, F, device="cuda", generator=g) * F ** -0.5).bfloat16()
    results = []
    for pair in (True, False):
        if not pair:
            monkeypatch.setattr(M, "_pair_tokens_pays", lambda *_: False)
        plan = M.GroupedPlan(idx, E, d, F)
        assert pair or not plan.on_pair
        results.append([(plan, plan.forward(M.FWD_GU, plan.gather(x), wgu)), (plan, plan.forward(M.FWD_DN, plan.gather(act), wd)),
                        (plan, plan.dgrad(M.DGRAD_DN, plan.gather(dout), wd)), (plan, plan.dgrad(M.DGRAD_GU, plan.gather(dy), wgu))])
    ops.check_status(torch.device("cuda"))
    e = idx[:, 0].long()
    for (a, w, back), (plan, got), (_, old) in zip(((x, wgu, False), (act, wd, False), (dout, wd, True), (dy, wgu, True)), *results):
        wide = w.double().view(E, -1, w.shape[1])
        if back:
            wide = wide.transpose(1, 2)
        want = torch.zeros(T, wide.shape[1], dtype=torch.float64, device="cuda")
        for i in range(E):
            want[e == i] = a[e == i].double() @ wide[i].t()
        mine = got[plan.row_of.long()].double()
        assert ((mine - want).abs() <= want.abs() * 2.0 ** -8 + 1e-5 * want.abs().max()).all()      # one rounding, fp32 sums
        assert (mine - want).norm() <= 1.02 * (old[plan.row_of.long()].double() - want).norm()
        used = int(plan.offsets[E])
        assert (got[:used][plan.src_of[:used] < 0] == 0).all()          # padding rows
