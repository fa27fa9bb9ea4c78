"""Every launch shape that a simulation reports can be asked for again, for the
library's own choices and a caller's; above 12 warps only the library's own choice
is accepted, and is the same shape."""
import pytest

from chromo_gb300 import _native as nat

pytestmark = pytest.mark.gpu


def _shape(R, W, G, fp64):
    sim = nat.Sim([20] * R, [(3, 3, 3)] * R, 1, pos_fp64=fp64, warps_per_block=W, lanes_per_move=G)
    try:
        return sim.launch_shape()
    finally:
        sim.close()


@pytest.mark.parametrize("R", [1, 160, 310, 1300])
@pytest.mark.parametrize("W,G,fp64", [(0, 0, False), (0, 16, False), (0, 8, False), (0, 0, True), (5, 32, False),
                                      (12, 16, False), (12, 32, True)])
def test_reported_shape_is_accepted(R, W, G, fp64):
    got = _shape(R, W, G, fp64)
    again = _shape(R, got[0], got[1], fp64)
    assert again[:2] == got[:2]
    if W > 0 or got[0] > 12 or fp64 or got[1] != 32:
        assert again == got


def test_other_shapes_above_twelve_warps_are_refused():
    own = _shape(1, 0, 32, False)[0]
    assert own > 12
    for W in (13, 14, 15, 17, -1):
        with pytest.raises(nat.CgError):
            _shape(1, W, 32, False)
    for R, W, fp64 in ((160, 16, False), (1, 16, True)):
        with pytest.raises(nat.CgError):
            _shape(R, W, 32, fp64)
