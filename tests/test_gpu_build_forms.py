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
