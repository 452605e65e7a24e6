"""The one-SM form of the per-trajectory kernel (FP64, fixed RK4 steps) against the general
form, which SAVE_TRAJECT runs take, and against the oracle (coupled states, AT-MQCT), on
linear-rotor tables of 1 to 441 states: one state, rows that end inside a warp, more threads
than the wide register split holds, the last size that fits one SM and the first that does not.

Tolerance: the two forms differ by the order of their sums (at most 441 terms, 2e-16 each) in
up to 2 000 right-hand sides, which enter each result with weights of order one and the
back-reaction's growth (below 100): 441^(1/2) * 2e-16 * 2000 * 100 < 1e-9."""
import numpy as np
import pytest

from mqct_b200 import synthetic as syn
from test_gpu_propagate import _straight_path

pytestmark = pytest.mark.gpu
TOL = 1e-9
E0 = 700.0 * syn.CM_TO_HARTREE


def _tables(mq, jmax, r_last=20.0, seed=3):
    s = mq.CollisionSystem(1, [(j,) for j in range(jmax + 1)], BE=1.93)
    R = mq.r_grid(60, 4.0, r_last)
    g = np.random.default_rng(seed)
    diag = s.ind_mat[:, 0] == s.ind_mat[:, 1]
    c = np.where(diag, 1.0, 0.0) + 0.5 * g.uniform(-1, 1, s.P) / (jmax + 1)
    mat = c[:, None] * (2e-2 * np.exp(-(R - 4.0) / 0.9) - 4e-4 * (6.0 / R) ** 6)
    return mq.PropagationTables.from_system(s, R, mat, 6.0)


def _oracle_tables(oracle, tab):
    return oracle.OracleTables(tab.j12, tab.m12, tab.ej, tab.ind_mat, tab.R, tab.mat, tab.y2,
                               tab.mass_au)


def _batch(mq, tab, n=12, **kw):
    """Impact parameters from head-on to beyond the start (the last, skipped), several initial
    states, one step cap and one time limit."""
    k = np.sqrt(2 * tab.mass_au * E0)
    tr = [mq.Trajectory(E0 * (1 + 0.05 * i), float(1.5 * i * k), 1 + (7 * i) % tab.n_states, 40.0,
                        16.0, 17.0) for i in range(n)]
    tr[-1].l_real = float(18.0 * np.sqrt(2 * tab.mass_au * tr[-1].e_coll))
    tr[1].max_steps = 50
    tr[2].time_lim = 5000.0
    return tr


@pytest.mark.parametrize("jmax,r_last", [(0, 20.0), (4, 20.0), (7, 12.0), (11, 20.0), (19, 20.0),
                                         (20, 20.0)])
def test_matches_general_form(mq, gpu_available, jmax, r_last):
    tab = _tables(mq, jmax, r_last)
    trajs = _batch(mq, tab)
    amp, cls, diag = mq.propagate(tab, trajs, arith=mq.PROP_FP64)
    a0, c0, d0, _ = mq.propagate_record(tab, trajs)
    assert set(d0[:, 4]) == {0.0, 1.0, 2.0}
    assert np.array_equal(diag[:, [1, 4, 5, 6]], d0[:, [1, 4, 5, 6]])
    assert np.max(np.abs(amp - a0)) < TOL
    assert np.allclose(cls, c0, rtol=TOL, atol=TOL)
    assert np.allclose(diag, d0, rtol=TOL, atol=TOL)


@pytest.mark.parametrize("cs", [False, True])
def test_shared_cta_equals_single_runs(mq, gpu_available, cs):
    """More trajectories than CTAs, of several initial m-blocks: each as if run alone."""
    tab = _tables(mq, 6)
    trajs = _batch(mq, tab) * 120
    plan = mq.PropagationPlan(tab, arith=mq.PROP_FP64)
    plan.set_coupled_states(cs)
    amp, cls, diag = plan.run(trajs)
    for i in range(12):
        a, c, d = plan.run(trajs[i:i + 1])
        for x, y in ((amp, a), (cls, c), (diag, d)):
            assert np.array_equal(x[i::12], np.repeat(y, 120, axis=0))
    plan.close()


@pytest.mark.parametrize("jmax", [0, 5, 19, 24])
def test_coupled_states(mq, oracle, gpu_available, jmax):
    tab = _tables(mq, jmax)
    trajs = _batch(mq, tab, 8)
    amp, cls, diag = mq.propagate(tab, trajs, arith=mq.PROP_FP64, coupled_states=True)
    ot = [oracle.make_traj(t.e_coll, t.l_real, t.s_st, t.dt, t.r_start, t.r_fin, t.numb_orb_prds,
                           t.numb_oscl_prds, t.time_lim, t.max_steps, cs=True) for t in trajs]
    oamp, ocls, odiag = oracle.propagate_batch(_oracle_tables(oracle, tab), ot)
    assert np.array_equal(diag[:, 1], odiag[:, 1])
    assert np.max(np.abs(amp - oamp)) < TOL
    assert np.allclose(cls[:, :2], ocls[:, :2], rtol=TOL, atol=TOL)


@pytest.mark.parametrize("jmax,dt", [(0, 40.0), (5, 17.0), (19, 40.0)])
def test_at_paths(mq, oracle, gpu_available, jmax, dt):
    """Paths of several lengths: the last step shortened, within one 16-step window, on its
    edge, and a path shorter than one step; a step cap; R beyond the last grid point."""
    tab = _tables(mq, jmax, 15.0)
    v = np.sqrt(2 * E0 / tab.mass_au)
    paths = [_straight_path(b, v, 18.0, tab.mass_au, n=900) for b in (4.5, 6.0, 9.0, 6.0, 5.0, 5.0)]
    for i, t_end in ((2, 16 * dt), (3, 15.5 * dt), (4, 0.6 * dt)):
        paths[i][:, 0] *= t_end / paths[i][-1, 0]
    trajs = [mq.Trajectory(E0, 0.0, 1, dt, 18.0, 18.0) for _ in paths]
    trajs[5].max_steps = 33
    amp, cls, diag = mq.propagate(tab, trajs, arith=mq.PROP_FP64, mode=mq.MODE_AT, at_paths=paths)
    otab = _oracle_tables(oracle, tab)
    for i, p in enumerate(paths):
        t = trajs[i]
        oamp, odiag = oracle.dotraject_at(otab, oracle.make_traj(
            E0, 0.0, 1, dt, 18.0, 18.0, max_steps=t.max_steps), p)
        assert diag[i, 1] == odiag[1] and diag[i, 4] == (1 if i == 5 else 0)
        assert abs(diag[i, 0] - odiag[0]) <= 1e-12 * odiag[0]
        assert np.max(np.abs(amp[i] - oamp)) < TOL
