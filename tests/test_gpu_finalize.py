"""The last step of every matrix build (cut-off and spline, one warp per element) and the
expansion contraction in front of it, at the edges of their register-resident forms: the
radial sizes where the form changes (128, 224, 352, 544 points), the smallest grids, few and
many pairs (groups of 8, 4, 2 and 1), terms in shared memory and not.

Tolerances: matrix elements 1e-12 of the largest element (FP64 sums of the same products as
the oracle's), y2 against the host's recurrence 1e-10 of the largest (FP64 recurrences of up
to 600 steps whose factors are below 1, composed in another order)."""
import numpy as np
import pytest

from mqct_b200 import synthetic as syn

pytestmark = pytest.mark.gpu


def _system(mq, j1, j2s):
    lv = syn.asym_channels(j1)
    return mq.CollisionSystem(8, [c + (j2,) for j2 in j2s for c in lv], A=27.88, B=9.28, C=14.52,
                              BE=60.853)


def _terms(lab, R, seed):
    rng = np.random.default_rng(seed)
    a, b = rng.normal(size=len(lab)) * 500.0, rng.uniform(0.5, 1.5, len(lab))
    return a * np.exp(-b * (R[:, None] - 5.0))


def _oracle(oracle, s, lab, T):
    ch = s.channels
    osys = oracle.OracleSystem(8, ch[:, 0], ch[:, 1], ch[:, 2], ch[:, 3], e_ch=s.e_ch,
                               vec1=s.vec1.reshape(-1), ldv=s.ldv)
    return oracle.expansion_matrix_type8(osys, osys.states(), s.ind_mat, lab, T)


def _check_y2(mq, R, m, y2):
    ref = mq.spline_y2(R, m) if len(R) >= 3 else np.zeros_like(m)
    assert np.max(np.abs(y2 - ref)) <= 1e-10 * max(np.abs(ref).max(), 1e-300)


@pytest.mark.parametrize("nR", [2, 3, 4, 31, 33, 34, 35, 96, 127, 128, 129, 162, 224, 225, 352,
                                353, 544, 545, 600])
def test_expansion_sizes(mq, oracle, gpu_available, nR):
    s = _system(mq, 2, (0, 2))
    lab = mq.expansion_terms_list(8, 4, 2, axl_sym1=2, equ_sym2=2)
    R = np.linspace(3.0, 20.0, nR)
    T = _terms(lab, R, nR)
    m, y2, sk = mq.build_matrix_expansion(s, R, lab, T, mij_cutoff=0.0)
    mo = _oracle(oracle, s, lab, T)
    assert np.max(np.abs(m - mo)) <= 1e-12 * np.abs(mo).max()
    _check_y2(mq, R, m, y2)
    assert not sk.any()


@pytest.mark.parametrize("nR,n_l1", [(50, 5), (200, 5), (101, 9), (300, 5)])
def test_expansion_many_pairs(mq, oracle, gpu_available, nR, n_l1):
    """Enough pairs for the widest groups; at (101, 9) the terms do not fit in shared memory."""
    s = _system(mq, 4, (0, 2))
    assert s.P > 37888
    lab = mq.expansion_terms_list(8, n_l1, 4, axl_sym1=1 if n_l1 > 5 else 2, equ_sym2=2)
    R = np.linspace(3.0, 20.0, nR)
    T = _terms(lab, R, nR)
    m, y2, sk = mq.build_matrix_expansion(s, R, lab, T, mij_cutoff=1e-6)
    mo = _oracle(oracle, s, lab, T)
    at = [np.argmin(np.abs(R - r)) for r in (6.0, 8.0)]
    drop = np.abs(mo[:, at]).max(axis=1) < 1e-6 * mq.CM_TO_HARTREE
    assert drop.any() and not drop.all()
    assert np.array_equal(sk.astype(bool), drop)
    mo[drop] = 0.0
    assert np.max(np.abs(m - mo)) <= 1e-12 * np.abs(mo).max()
    _check_y2(mq, R, m, y2)
    assert not m[drop].any() and not y2[drop].any()


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_expansion_non_finite_terms(mq, oracle, gpu_available, bad):
    """A term that is not finite reaches every element at its radial point (0 x inf is NaN),
    also those whose coefficient of the term is zero; the other points are untouched."""
    s = _system(mq, 2, (0, 2))
    lab = mq.expansion_terms_list(8, 4, 2, axl_sym1=2, equ_sym2=2)
    R = np.linspace(3.0, 20.0, 60)
    T = _terms(lab, R, 7)
    mo = _oracle(oracle, s, lab, T)
    T[41, 3] = bad
    m, _, _ = mq.build_matrix_expansion(s, R, lab, T, mij_cutoff=0.0)
    assert not np.isfinite(m[:, 41]).any()
    rest = np.arange(60) != 41
    assert np.max(np.abs(m[:, rest] - mo[:, rest])) <= 1e-12 * np.abs(mo).max()


@pytest.mark.parametrize("prec", ["PREC_FP64", "PREC_F16X3"])
@pytest.mark.parametrize("nR", [2, 3, 17, 128, 129, 225, 353, 545])
def test_build_spline_sizes(mq, gpu_available, nR, prec):
    """y2 of a direct build (one or several partial sums per element) is the spline of its
    Mat_el at every size of the finalize."""
    s = mq.CollisionSystem(4, syn.asym_channels(2), **dict(A=27.9, B=14.5, C=9.3))
    R = np.linspace(4.0, 20.0, nR)
    m, y2, sk = mq.build_matrix(s, R, (10, 9, 0, 0, 0, 0, 1), syn.site_pes(6, seed=4),
                                precision=getattr(mq, prec), mij_cutoff=0.0)
    assert np.abs(m).max() > 0 and not sk.any()
    _check_y2(mq, R, m, y2)


@pytest.mark.parametrize("jmax,nR,n_alpha", [(2, 31, 0), (2, 33, 3), (6, 33, 0), (6, 48, 0),
                                             (6, 100, 0), (6, 161, 2), (6, 300, 0), (8, 40, 0),
                                             (8, 81, 0)])
def test_build_fp64_tiles(mq, gpu_available, jmax, nR, n_alpha):
    """The FP64 contraction's tile shapes (chosen by the number of row tiles and R points),
    ragged columns and grid chunks: an element does not depend on the other radial points, so
    every third one agrees with a build of those points alone (another shape); 1e-13 of the
    largest, the two being the same FP64 products and order."""
    s = mq.CollisionSystem(4, syn.asym_channels(jmax), **dict(A=27.9, B=14.5, C=9.3))
    R = np.linspace(4.0, 20.0, nR)
    grid, pes = (9, 7, n_alpha, 0, 0, 0, 1), syn.site_pes(6, seed=4)
    m, _, _ = mq.build_matrix(s, R, grid, pes, mij_cutoff=0.0)
    m3, _, _ = mq.build_matrix(s, R[::3], grid, pes, mij_cutoff=0.0)
    assert np.max(np.abs(m[:, ::3] - m3)) <= 1e-13 * np.abs(m).max()
