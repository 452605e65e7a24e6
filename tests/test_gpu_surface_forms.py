"""Built-in surfaces in the forms that the weight kernels tell apart: distinct sites with several
terms each and in any order, beyond 512 terms, site surfaces of a diatom, Legendre surfaces of a
top and beyond 40 terms.

Tolerances.  FP64: a value of the surface sums at most 567 terms of both signs, whose rounding
(567 x 1.1e-16 = 6e-14 of the sum of magnitudes, below ten times the largest element) enters each
element through weights whose sum is of order one: 1e-11 of the largest element.  Split
precision: the bounds of the split-precision tests."""
import numpy as np
import pytest

from mqct_b200 import synthetic as syn
from test_gpu_tc import _errors

pytestmark = pytest.mark.gpu
TOP = dict(A=27.9, B=14.5, C=9.3)
PRECS = ["fp64", "f16x3", "bf16x3"]


def _prec(mq, name):
    return {"fp64": mq.PREC_FP64, "f16x3": mq.PREC_F16X3, "bf16x3": mq.PREC_BF16X3}[name]


def _split(pes, per, k, seed):
    """Every term as k terms that add up to it (depth and C6 shared out), in random order."""
    p = np.repeat(np.asarray(pes["params"], float).reshape(-1, per), k, axis=0)
    p[:, per - 5] /= k
    p[:, per - 2] /= k
    np.random.default_rng(seed).shuffle(p, axis=0)
    return dict(pes, n_terms=len(p), params=p.reshape(-1))


def _check(m, ref, prec):
    if prec == "fp64":
        assert np.max(np.abs(m - ref)) <= 1e-11 * np.max(np.abs(ref))
        return
    med, _, ek_med, ek_max = _errors(m, ref)
    if prec == "bf16x3":
        assert med < 5e-5, med
    else:
        assert ek_med < 5e-6 and ek_max < 5e-5, (ek_med, ek_max)


@pytest.mark.parametrize("prec", PRECS)
@pytest.mark.parametrize("k", [2, 6, 7])
def test_two_rotors_terms_of_a_site_pair(mq, gpu_available, k, prec):
    lv = syn.asym_channels(1)
    s = mq.CollisionSystem(0, [a + b for a in lv for b in lv], **TOP)
    R, grid, pes = mq.r_grid(12, 5.0, 12.0), (6, 4, 0, 5, 3, 4, 1), syn.site_pes2()
    ref = mq.build_matrix(s, R, grid, pes, precision=mq.PREC_FP64, mij_cutoff=0.0)[0]
    m = mq.build_matrix(s, R, grid, _split(pes, 7, k, k), precision=_prec(mq, prec), mij_cutoff=0.0)[0]
    _check(m, ref, prec)


@pytest.mark.parametrize("prec", PRECS)
@pytest.mark.parametrize("sys_type", [1, 4])
@pytest.mark.parametrize("k", [1, 3, 42, 43])
def test_rotor_and_atom_sites(mq, oracle, gpu_available, sys_type, k, prec):
    pes = _split(syn.site_pes(12, seed=3), 6, k, k)
    R = mq.r_grid(30, 4.0, 20.0)
    if sys_type == 1:
        s, grid = mq.CollisionSystem(1, [(j,) for j in range(4)], BE=1.93), (20, 0, 0, 0, 0, 0, 1)
    else:
        s, grid = mq.CollisionSystem(4, syn.asym_channels(2), **TOP), (12, 11, 0, 0, 0, 0, 1)
    m = mq.build_matrix(s, R, grid, pes, precision=_prec(mq, prec), mij_cutoff=0.0)[0]
    _check(m, _oracle(oracle, s, R, grid, pes), prec)


@pytest.mark.parametrize("prec", PRECS)
@pytest.mark.parametrize("sys_type", [1, 4])
@pytest.mark.parametrize("n", [1, 2, 40, 41])
def test_legendre(mq, oracle, gpu_available, n, sys_type, prec):
    pes = syn.legendre_pes(n, seed=n)
    R = mq.r_grid(130, 4.0, 20.0)
    if sys_type == 1:
        s, grid = mq.CollisionSystem(1, [(j,) for j in range(5)], BE=1.93), (33, 0, 0, 0, 0, 0, 1)
    else:
        s, grid = mq.CollisionSystem(4, syn.asym_channels(1), **TOP), (17, 9, 0, 0, 0, 0, 1)
    m = mq.build_matrix(s, R, grid, pes, precision=_prec(mq, prec), mij_cutoff=0.0)[0]
    _check(m, _oracle(oracle, s, R, grid, pes), prec)


def _oracle(oracle, s, R, grid, pes):
    ch = s.channels
    cols = (ch[:, 0],) if s.sys_type == 1 else (ch[:, 0], ch[:, 1], ch[:, 2])
    vec = np.ones(s.n_channels) if s.sys_type == 1 else s.vec1.reshape(-1)
    osys = oracle.OracleSystem(s.sys_type, *cols, e_ch=s.e_ch, vec1=vec,
                               ldv=1 if s.sys_type == 1 else s.ldv)
    opes = oracle.OraclePes(pes["kind"], pes["n_terms"], pes["params"], sites1=pes["sites1"])
    return oracle.build_matrix(osys, osys.states(), s.ind_mat, R, grid, opes, mij_cut=0.0)[0]
