"""What jenhine_b200/motion.py refuses: a motion that is not one row of (at
least) six numbers, fewer motions than views, no views."""
import numpy as np
import pytest

from jenhine_b200.motion import moved_ptms, ptm_derivatives, rigid


@pytest.mark.parametrize("shape,error", [((), IndexError), ((0,), IndexError), ((5,), IndexError), ((1, 6), IndexError),
                                         ((2, 6), IndexError), ((6, 1), ValueError), ((6, 6), ValueError)])
def test_rigid_refuses_what_is_not_one_motion(shape, error):
    with pytest.raises(error):
        rigid(np.ones(shape))


def test_rigid_reads_six_numbers():
    t = np.arange(7.0)
    for a, b in zip(rigid(t), rigid(t[:6])):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("f", [moved_ptms, ptm_derivatives])
def test_views_and_motions(f):
    P = np.random.default_rng(0).standard_normal((4, 12))
    with pytest.raises(ValueError):
        f(P[:0], np.ones((0, 6)))
    with pytest.raises(ValueError):
        f(P[:0], np.ones((3, 6)))
    with pytest.raises(IndexError):
        f(P, np.ones((3, 6)))
    np.testing.assert_array_equal(f(P, np.ones((6, 6))), f(P, np.ones((4, 6))))
