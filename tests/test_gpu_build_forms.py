"""Matrix builds at inputs where a form of the build could go wrong: channels that no state uses.
Results are compared with the same build without what should not matter, bit for bit."""
import numpy as np
import pytest

from mqct_b200 import synthetic as syn

pytestmark = pytest.mark.gpu
TOP = dict(A=27.9, B=14.5, C=9.3)
GRID5 = (6, 4, 0, 5, 3, 4, 1)


def _two_tops(mq):
    lv = syn.asym_channels(1)
    return mq.CollisionSystem(0, [a + b for a in lv for b in lv], **TOP)


def _with_unused_channel(s, j1, j2):
    """The system with one more channel, the last one, that has no states."""
    s.n_channels += 1
    for name, v in (("j1", j1), ("ka1", 0), ("kc1", 0), ("j2", j2), ("ka2", 0), ("kc2", 0)):
        old = getattr(s, name)
        setattr(s, name, np.append(old if len(old) == s.n_channels - 1 else np.zeros(s.n_channels - 1),
                                   v).astype(np.int32))
    s.vec1, s.vec2 = (np.vstack([v, np.zeros((1, s.ldv))]) for v in (s.vec1, s.vec2))
    return s


@pytest.mark.parametrize("j1,j2", [(20, 0), (0, 20), (20, 20), (-1, -1)])
def test_unused_channel_of_two_rotors(mq, gpu_available, j1, j2):
    """A channel without states is not read: its j may be beyond its row of vector values."""
    R, pes = mq.r_grid(12, 5.0, 12.0), syn.site_pes2()
    ref = mq.build_matrix(_two_tops(mq), R, GRID5, pes, mij_cutoff=0.0)
    out = mq.build_matrix(_with_unused_channel(_two_tops(mq), j1, j2), R, GRID5, pes, mij_cutoff=0.0)
    for a, b in zip(out, ref):
        assert np.array_equal(a, b)


def test_unused_channel_of_a_top(mq, gpu_available):
    """Its j may be beyond the rotor functions' table of factorials."""
    R, pes = mq.r_grid(12, 5.0, 12.0), syn.site_pes(6, seed=4)
    top = lambda: mq.CollisionSystem(4, syn.asym_channels(2), **TOP)  # noqa: E731
    ref = mq.build_matrix(top(), R, (9, 7, 0, 0, 0, 0, 1), pes, mij_cutoff=0.0)
    out = mq.build_matrix(_with_unused_channel(top(), 80, 0), R, (9, 7, 0, 0, 0, 0, 1), pes,
                          mij_cutoff=0.0)
    for a, b in zip(out, ref):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("nR", [3, 33, 70, 201])
@pytest.mark.parametrize("nb,ng", [(3, 5), (4, 4), (9, 7)])
@pytest.mark.parametrize("n_alpha", [1, 2, 3, 48])
def test_fp64_alpha_axis(mq, gpu_available, n_alpha, nb, ng, nR):
    """The alpha axis as a grid against its analytic 2 pi, at less than one chunk of grid points,
    one chunk, and four with a remainder, and in every tile shape.  A sum of at most 63 x 48 terms
    in FP64 is off by 3 024 x 1.1e-16 = 3.4e-13 of the sum of their magnitudes, which the
    largest element exceeds to within a factor of ten: 1e-11 of it bounds the difference."""
    s = mq.CollisionSystem(4, syn.asym_channels(3), **TOP)
    R, pes = mq.r_grid(nR, 3.0, 25.0), syn.site_pes(6, seed=5)
    kw = dict(precision=mq.PREC_FP64, mij_cutoff=0.0)
    ref = mq.build_matrix(s, R, (nb, ng, 0, 0, 0, 0, 1), pes, **kw)[0]
    out = mq.build_matrix(s, R, (nb, ng, n_alpha, 0, 0, 0, 1), pes, **kw)[0]
    assert np.max(np.abs(out - ref)) <= 1e-11 * np.max(np.abs(ref))
