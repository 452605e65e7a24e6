"""The grouping of pairs in the expansion build: results do not depend on it, bit for bit."""
import copy

import numpy as np
import pytest
import torch

from mqct_b200 import synthetic as syn

pytestmark = pytest.mark.gpu
TOP = dict(A=27.88, B=9.28, C=14.52)


def _terms(n, R, seed=1):
    g = np.random.default_rng(seed)
    a, b = g.uniform(-4000.0, 4000.0, n), g.uniform(1.2, 2.0, n)
    return a[:, None] * np.exp(-b[:, None] * (R - 5.0)) - g.uniform(-1e5, 1e5, n)[:, None] / R ** 6


def _run(mq, s, R, lab, T, pairs=slice(None), times=1):
    s = copy.copy(s)
    s.ind_mat = np.ascontiguousarray(s.ind_mat[pairs])
    s.P = len(s.ind_mat)
    plan = mq.ExpansionPlan(s, R, lab, mij_cutoff=1e-6)
    t = torch.from_numpy(T).cuda()
    out = []
    for _ in range(times):
        m = torch.zeros((s.P, len(R)), dtype=torch.float64, device="cuda")
        y, k = torch.zeros_like(m), torch.zeros(s.P, dtype=torch.int32, device="cuda")
        plan.execute(t, m, y, k)
        plan.sync()
        out.append([x.cpu().numpy() for x in (m, y, k)])
    plan.close()
    for o in out[1:]:  # a plan's later runs start from the group queue that the first one left
        assert all(np.array_equal(x, z) for x, z in zip(o, out[0]))
    return out[0]


@pytest.mark.parametrize("jmax,nR", [(9, 101), (9, 128), (8, 129), (8, 224), (8, 225)])
def test_stored_coefficients_in_groups(mq, gpu_available, jmax, nR):
    """Asymmetric top + atom: eight, four and two pairs to a warp, more groups than warps, against
    builds of 5 000 pairs each, which take two."""
    s = mq.CollisionSystem(4, syn.asym_channels(jmax), **TOP)
    R = mq.r_grid(nR, 4.0, 30.0)
    lab = [(l, m) for l in range(6) for m in range(0, l + 1, 2)]
    T = _terms(len(lab), R)
    whole = _run(mq, s, R, lab, T, times=3)
    assert 0 < np.count_nonzero(whole[2]) < s.P
    for p0 in range(0, s.P, 5000):
        part = _run(mq, s, R, lab, T, slice(p0, p0 + 5000))
        assert all(np.array_equal(x[p0:p0 + 5000], z) for x, z in zip(whole, part))


@pytest.mark.parametrize("sys_type", [1, 8])
@pytest.mark.parametrize("nR", [101, 600])
def test_channels_beyond_32_bit_pair_counts(mq, gpu_available, sys_type, nR):
    """46 341 channels, of which a few have states: their pairs do not fit a 32-bit count."""
    R = mq.r_grid(nR, 4.0, 30.0)
    if sys_type == 1:
        s = mq.CollisionSystem(1, [(j,) for j in range(6)], BE=1.93)
        lab, cols = [(l,) for l in range(5)], ("j1",)
    else:
        s = mq.CollisionSystem(8, [c + (0,) for c in syn.asym_channels(1)], BE=60.853, **TOP)
        lab, cols = [(2, 0, 0, 2)], ("j1", "ka1", "kc1", "j2")
    T = _terms(len(lab), R)
    ref = _run(mq, s, R, lab, T)
    big = copy.copy(s)
    more = 46341 - s.n_channels
    big.n_channels = 46341
    for c in cols:
        setattr(big, c, np.append(getattr(s, c), np.zeros(more)).astype(np.int32))
    if s.vec1 is not None:
        big.vec1 = np.vstack([s.vec1.reshape(s.n_channels, -1), np.zeros((more, s.ldv))])
    assert np.any(ref[0])
    assert all(np.array_equal(x, z) for x, z in zip(_run(mq, big, R, lab, T), ref))
