"""The cluster-resident engine where a right-hand side's point matters at once: trajectories
that start inside the interaction region and are cut off after 40 RK4 steps, from their start
(MQCT_ENGINE_RESIDENT) and handed over by the lockstep engine after its first graph of 64
rounds (MQCT_ENGINE_LOCKSTEP_TAIL), against the FP32 per-trajectory kernel.

Amplitudes within 5e-5: 160 right-hand sides whose FP32 inputs and products round to 6e-8,
a few of them adding up in each."""
import numpy as np
import pytest

from test_gpu_lockstep import c2_tables  # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("engine,cluster", [("ENGINE_RESIDENT", 0), ("ENGINE_RESIDENT", 8),
                                            ("ENGINE_LOCKSTEP_TAIL", 0)])
@pytest.mark.parametrize("r0", [5.5, 7.25])
def test_short_runs_in_the_interaction_region(mq, gpu_available, c2_tables, engine, cluster, r0):
    tab = c2_tables["tab"]
    near = [t for t in c2_tables["trajs"]
            if t.l_real + 1.0 < 0.6 * r0 * np.sqrt(2 * tab.mass_au * t.e_coll)][:20]
    assert len(near) >= 10
    trajs = [mq.Trajectory(t.e_coll, t.l_real, t.s_st, t.dt, r0, 25.0, max_steps=40) for t in near]
    out = {}
    for e in (engine, "ENGINE_PER_TRAJECTORY"):
        plan = mq.PropagationPlan(tab, mq.PROP_FP32)
        plan.set_engine(getattr(mq, e))
        if cluster:
            plan.set_cluster(cluster)
        out[e] = plan.run(trajs)
        assert plan.engine()[0] == getattr(mq, e)
        if e == "ENGINE_LOCKSTEP_TAIL":
            assert plan.handed() == len(trajs)
        plan.close()
    (a, c, d), (a0, c0, d0) = out[engine], out["ENGINE_PER_TRAJECTORY"]
    assert np.max(np.abs(a - a0)) < 5e-5
    assert np.array_equal(d[:, 4], d0[:, 4]) and np.array_equal(d[:, 1], d0[:, 1])
    assert np.allclose(c, c0, rtol=5e-5, atol=5e-5)
