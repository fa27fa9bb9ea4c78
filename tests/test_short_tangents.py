"""Short tangent rotations (groups of 8 or 16 lanes, bead hash) at the edges of
their range -- one bead, a group's lanes, twice them, one more -- on chains so
short that most moves redraw beads and conflict, and on longer ones: the state
equals that of the path of list comparisons (8 lanes per move) bit for bit."""
import numpy as np
import pytest

from chromo_gb300 import _native as nat
from chromo_gb300 import synthetic as syn
from chromo_gb300.device import binding_params, bonds_array, field_params, move_ctl
from chromo_gb300.energetics import dss_parameters

pytestmark = pytest.mark.gpu


def _run(n, amp, twist, W, G):
    rng = np.random.default_rng(n)
    r = syn.gaussian_walk(rng, n, 16.5)
    t3, t2 = syn.tangents_from_coordinates(r)
    _, eb, g, ep, epp, eta = dss_parameters(np.full(n - 1, 16.5), 53.0)
    sim = nat.Sim([n], [(6, 6, 6)], 1, max_tangent=n, warps_per_block=W, lanes_per_move=G)
    sim.set_chain(0, r=r, t3=t3, t2=t2, states=np.zeros((n, 1), np.int64), marks=np.zeros((n, 1), np.int64),
                  bonds=bonds_array(eb, g, ep, epp, eta))
    if twist:
        sim.set_twist(0, np.full(n - 1, 6.0), np.full(n - 1, 16.5 * 2 * np.pi / 10.5 / 0.332))
    sim.set_field(0, field_params(field_kind=2, nxyz=(6, 6, 6), widths=(240.0,) * 3, n_binders=1, bead_vol=523.6,
                                  pref=[0.0], intra=[0.0]))
    sim.set_binding(0, binding_params(sites=[2], e_mod=[0.0], e_nomod=[0.0], mu=[0.0]))
    sim.set_controllers(0, [move_ctl("tangent_rotation", amp_move=0.3, amp_bead=amp, num_per_cycle=61, simple=False)])
    sim.deposit(-1)
    sim.run(12, 5)
    sim.sync()
    out = sim.get_chain(0) + (sim.tally(0), np.array([c.acc_rate for c in sim.get_controllers(0)]))
    sim.close()
    return out


@pytest.mark.parametrize("twist", [False, True])
@pytest.mark.parametrize("n,amp", [(2, 1), (2, 2), (9, 8), (9, 9), (17, 16), (18, 17), (33, 32), (34, 33), (40, 15),
                                   (300, 7), (300, 31), (3000, 16), (3000, 32)])
def test_short_tangents_equal_list_path(n, amp, twist):
    want = _run(n, amp, twist, 2, 8)
    assert want[-2][3, 1] > 0  # rotations were accepted
    for W in (1, 6, 12):
        for a, b in zip(want, _run(n, amp, twist, W, 32)):
            np.testing.assert_array_equal(a, b)
