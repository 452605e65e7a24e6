"""The tcgen05 contraction where its splits and column shares change: few tiles over a long grid
(more K ranges than waves need), column parts of 16 to 112 and just above, both epilogue layouts,
1 to 5 alpha points; and surfaces that are not finite.  Tolerances: those of the split-precision
tests (16 and 22 bits kept of either operand)."""
import numpy as np
import pytest

from mqct_b200 import synthetic as syn
from test_gpu_tc import _c2_small, _errors

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nR,n_alpha,warps", [(16, 0, 8), (104, 0, 16), (112, 5, 16), (113, 4, 8),
                                              (200, 0, 8)])
@pytest.mark.parametrize("prec", ["bf16x3", "f16x3"])
def test_many_ranges_and_parts(mq, gpu_available, nR, n_alpha, warps, prec):
    import torch
    s = _c2_small(mq, 2)
    R = mq.r_grid(nR, 3.0, 25.0)
    grid, pes = (40, 40, n_alpha, 0, 0, 0, 1), syn.site_pes(12, seed=2)
    m64, _, _ = mq.build_matrix(s, R, grid, pes, precision=mq.PREC_FP64, mij_cutoff=0.0)
    plan = mq.MatrixPlan(s, R, grid, pes, mij_cutoff=0.0,
                         precision=mq.PREC_BF16X3 if prec == "bf16x3" else mq.PREC_F16X3)
    assert plan.layout()[1] > 4
    plan.set_epilogue(warps)
    d = torch.empty((s.P, nR), dtype=torch.float64, device="cuda")
    for _ in range(2):
        plan.execute(d.data_ptr())
        plan.sync()
    m3 = d.cpu().numpy()
    plan.close()
    med, _, ek_med, ek_max = _errors(m3, m64)
    if prec == "bf16x3":
        assert med < 5e-5, med
    else:
        assert ek_med < 5e-6 and ek_max < 5e-5, (ek_med, ek_max)


@pytest.mark.parametrize("prec", ["bf16x3", "f16x3"])
def test_surface_not_finite(mq, gpu_available, prec):
    s = _c2_small(mq, 1)
    R = mq.r_grid(20, 3.0, 25.0)
    pes = syn.site_pes(12, seed=2)
    pes = dict(pes, params=np.array(pes["params"], float).copy())
    pes["params"].reshape(-1, 6)[:, 1] = np.nan  # the well depths
    m, _, _ = mq.build_matrix(s, R, (8, 8, 0, 0, 0, 0, 1), pes, mij_cutoff=0.0,
                              precision=mq.PREC_BF16X3 if prec == "bf16x3" else mq.PREC_F16X3)
    assert not np.isfinite(m).any()
