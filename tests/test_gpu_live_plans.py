"""Two live plans of different sizes: the second does not take from the first the shared memory
that its kernels ask for.  Results are compared with a plan that ran alone, bit for bit."""
import numpy as np
import pytest
import torch

from mqct_b200 import synthetic as syn
from test_gpu_onecta import _batch, _tables

pytestmark = pytest.mark.gpu


def _matrix_plan(mq, jmax, prec):
    s = mq.CollisionSystem(4, syn.asym_channels(jmax), A=27.9, B=14.5, C=9.3)
    R = mq.r_grid(112, 3.0, 25.0)
    plan = mq.MatrixPlan(s, R, (10, 9, 0, 0, 0, 0, 1), syn.site_pes(6, seed=2), precision=prec,
                         mij_cutoff=0.0)
    return plan, (s.P, len(R))


def _execute(plan, shape):
    out = torch.zeros(shape, dtype=torch.float64, device="cuda")
    plan.execute(out.data_ptr())
    plan.sync()
    return out.cpu().numpy()


@pytest.mark.parametrize("prec", ["FP64", "F16X3", "BF16X3"])
def test_matrix_plans(mq, gpu_available, prec):
    prec = getattr(mq, "PREC_" + prec)
    big, big_shape = _matrix_plan(mq, 7, prec)
    alone = _execute(big, big_shape)
    small, small_shape = _matrix_plan(mq, 2, prec)
    _execute(small, small_shape)
    assert np.array_equal(_execute(big, big_shape), alone)


@pytest.mark.parametrize("integrator", [None, ("ODEINT", 1e-6, 0.0)])
def test_propagation_plans(mq, gpu_available, integrator):
    """441 states in FP64 (beyond the one-SM form) and 9 states."""
    tabs = [_tables(mq, 20), _tables(mq, 2)]
    plans = [mq.PropagationPlan(t, arith=mq.PROP_FP64) for t in tabs]
    trajs = [_batch(mq, t, 4) for t in tabs]
    for tr in trajs[0] + trajs[1]:
        tr.time_lim = 2000.0
    plans[0].set_integrator(integrator)
    alone = plans[0].run(trajs[0])
    if integrator is None:
        plans[1].set_engine(mq.ENGINE_PER_TRAJECTORY)
    plans[1].set_integrator(integrator)
    plans[1].run(trajs[1])
    for a, b in zip(plans[0].run(trajs[0]), alone):
        assert np.array_equal(a, b)
    for p in plans:
        p.close()
