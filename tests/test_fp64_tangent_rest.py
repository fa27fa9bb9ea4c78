"""FP64 tangent rotations whose beads beyond a multiple of 32 go four lanes a bead (up
to 16 of them) or a lane each (more): as in test_fp64_tangents.py, equal to a lane
each throughout bit for bit, with many remainders on both sides of the line."""
import numpy as np
import pytest

from test_fp64_tangents import _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,amp", [(17, 17), (49, 49), (600, 17), (600, 50), (600, 300)])
def test_remainders(n, amp):
    want = _run(n, amp, 4, False)
    assert want[4][3, 1] > 0  # rotations were accepted
    for W in (1, 12):
        for a, b in zip(want, _run(n, amp, W, True)):
            np.testing.assert_array_equal(a, b)
