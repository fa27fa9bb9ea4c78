"""Tangent rotations on both sides of the line between the paths of 16 and of 32 lanes at the
default shape, for short chains and for up to 32 beads of long ones, against one move at a
time."""
import numpy as np
import pytest

from chromo_gb300 import workloads as wl
from chromo_gb300.device import move_ctl
from test_short_tangents import _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,amp", [(12, 8), (12, 9), (100, 13), (100, 14), (500, 17), (500, 18), (6000, 17), (6000, 24), (6000, 32), (6000, 33)])
def test_rotations_equal_one_at_a_time(n, amp):
    w = wl.Workload("long", np.array([n]), 10, 1, np.zeros((1, 1)), np.ones(1), [-4.0], [{}], 20, 0, amp)
    chains = wl.make_chains(w)
    out = []
    for W in (0, 1):
        sim = wl.build_sim(w, chains, warps_per_block=W)
        sim.set_controllers(0, [move_ctl("tangent_rotation", amp_move=0.4, amp_bead=amp, num_per_cycle=150, simple=False,
                                         bead_bounds=(1, n), move_bounds=(0.0, 1.0), acc_rate=0.5)])
        sim.run(2, 11)
        sim.sync()
        assert sim.tally(0)[3, 1] > 0
        out.append(sim.get_chain(0) + (sim.tally(0),))
        sim.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("n,amp", [(16, 16), (20, 17), (20, 18), (64, 32), (63, 32)])
def test_twisted_rotations_equal_eight_lanes(n, amp):
    want = _run(n, amp, True, 2, 8)
    assert want[-2][3, 1] > 0
    for a, b in zip(want, _run(n, amp, True, 0, 32)):
        np.testing.assert_array_equal(a, b)
