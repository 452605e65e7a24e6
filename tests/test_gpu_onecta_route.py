"""Which FP64 runs take the one-SM form of the per-trajectory kernel, and its AT-mode outputs."""
import numpy as np
import pytest

from test_gpu_onecta import E0, TOL, _batch, _oracle_tables, _tables
from test_gpu_propagate import _straight_path

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("jmax,fits", [(0, True), (4, True), (11, True), (19, True), (20, False),
                                       (24, False)])
@pytest.mark.parametrize("cs", [False, True])
def test_form_of_a_run(mq, gpu_available, jmax, fits, cs):
    tab = _tables(mq, jmax)
    trajs = _batch(mq, tab, 4)
    for t in trajs:
        t.max_steps = 20
    plan = mq.PropagationPlan(tab, arith=mq.PROP_FP64)
    assert not plan.one_sm()
    plan.set_coupled_states(cs)
    plan.run(trajs)
    assert plan.engine()[0] == mq.ENGINE_PER_TRAJECTORY and plan.one_sm() == fits
    for t in trajs:
        t.time_lim = 200.0
    plan.set_integrator(("ODEINT", 1e-6, 0.0))
    plan.run(trajs)
    assert not plan.one_sm()
    plan.set_integrator(None)
    plan.run(trajs)
    assert plan.one_sm() == fits
    if jmax == 4 and not cs:
        plan.set_engine(mq.ENGINE_LOCKSTEP)
        plan.run(trajs)
        assert plan.engine()[0] == mq.ENGINE_LOCKSTEP and not plan.one_sm()
    plan.close()
    single = mq.PropagationPlan(tab, arith=mq.PROP_FP32)
    single.run(trajs)
    assert not single.one_sm()
    single.close()


@pytest.mark.parametrize("jmax", [0, 5, 19])
def test_at_outputs(mq, oracle, gpu_available, jmax):
    """An AT run has no classical state, no energy balance and no coupling energy to report."""
    tab = _tables(mq, jmax)
    v = np.sqrt(2 * E0 / tab.mass_au)
    paths = [_straight_path(b, v, 18.0, tab.mass_au, n=300) for b in (4.5, 9.0)]
    trajs = [mq.Trajectory(E0, 0.0, 1, 40.0, 18.0, 18.0) for _ in paths]
    _, cls, diag = mq.propagate(tab, trajs, arith=mq.PROP_FP64, mode=mq.MODE_AT, at_paths=paths)
    assert np.all(cls == 0.0) and np.all(diag[:, [3, 5, 6, 7]] == 0.0)
    for i, p in enumerate(paths):
        _, od = oracle.dotraject_at(_oracle_tables(oracle, tab),
                                    oracle.make_traj(E0, 0.0, 1, 40.0, 18.0, 18.0), p)
        assert abs(diag[i, 2] - od[2]) < TOL
