"""Tangent rotations on both sides of the lines between the short path (a group of 8
or 16 lanes, beads in a hash) and the path of 32 lanes: by amplitude, and by the
chain's length for the amplitude, with and without twist.  The state equals that of
8 lanes per move bit for bit."""
import numpy as np
import pytest

from test_short_tangents import _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,amp,twist", [
    (12, 3, False), (11, 3, False), (342, 16, False), (341, 16, False), (2000, 16, False), (2000, 17, False),
    (8, 8, True), (10, 9, True), (128, 32, True), (127, 32, True), (2000, 32, True), (2000, 33, True)])
def test_both_sides_of_the_short_path(n, amp, twist):
    want = _run(n, amp, twist, 2, 8)
    assert want[-2][3, 1] > 0  # rotations were accepted
    for W in (0, 1, 12):
        for a, b in zip(want, _run(n, amp, twist, W, 32)):
            np.testing.assert_array_equal(a, b)
