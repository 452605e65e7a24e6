"""The FP32-pair sums of the tcgen05 contraction beyond their range: a sum over the alpha axis that
overflows FP32 is infinite, as a single partial sum that does."""
import numpy as np
import pytest
import torch

from mqct_b200 import synthetic as syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("warps", [8, 16])
def test_overflow_stays_infinite(mq, gpu_available, warps, sign):
    """V = 2e38 everywhere, 48 alpha points: a diagonal element's partial sum of two points is
    V / pi = 6e37, the sum of all 1.5e39."""
    s = mq.CollisionSystem(4, syn.asym_channels(1), A=27.9, B=14.5, C=9.3)
    R = mq.r_grid(20, 3.0, 25.0)
    pes = dict(kind=syn.PES_LEGENDRE, n_terms=1, params=np.array([sign * 2e38, 0.0, 0.0]),
               sites1=None, sites2=None)
    plan = mq.MatrixPlan(s, R, (8, 8, 48, 0, 0, 0, 1), pes, precision=mq.PREC_BF16X3, mij_cutoff=0.0)
    plan.set_epilogue(warps)
    d = torch.zeros((s.P, len(R)), dtype=torch.float64, device="cuda")
    plan.execute(d.data_ptr())
    plan.sync()
    m = d.cpu().numpy()
    diag = s.ind_mat[:, 0] == s.ind_mat[:, 1]
    assert np.all(m[diag] == sign * np.inf)
    assert not np.isnan(m).any()
