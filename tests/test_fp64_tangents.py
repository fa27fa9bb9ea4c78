"""FP64 storage: tangent rotations with four lanes a bead (passes of 8 beads) equal
the form of one lane a bead bit for bit, at the edges of the passes.  The latter
serves SSTWLC chains; a twist modulus of 1e-300 adds nothing to their energies."""
import numpy as np
import pytest

from chromo_gb300 import _native as nat
from chromo_gb300 import synthetic as syn
from chromo_gb300.device import binding_params, bonds_array, field_params, move_ctl
from chromo_gb300.energetics import dss_parameters

pytestmark = pytest.mark.gpu


def _run(n, amp, W, lanes):
    rng = np.random.default_rng(n)
    r = syn.gaussian_walk(rng, n, 16.5)
    t3, t2 = syn.tangents_from_coordinates(r)
    _, eb, g, ep, epp, eta = dss_parameters(np.full(n - 1, 16.5), 53.0)
    sim = nat.Sim([n], [(6, 6, 6)], 1, pos_fp64=True, max_tangent=n, warps_per_block=W)
    sim.set_chain(0, r=r, t3=t3, t2=t2, states=np.zeros((n, 1), np.int64), marks=np.zeros((n, 1), np.int64),
                  bonds=bonds_array(eb, g, ep, epp, eta))
    if not lanes:
        sim.set_twist(0, np.full(n - 1, 1e-300), np.zeros(n - 1))  # must be positive
    sim.set_field(0, field_params(field_kind=2, nxyz=(6, 6, 6), widths=(240.0,) * 3, n_binders=1, bead_vol=523.6,
                                  pref=[0.0], intra=[0.0]))
    sim.set_binding(0, binding_params(sites=[2], e_mod=[0.0], e_nomod=[0.0], mu=[0.0]))
    # position moves too: the boundary bonds' energies before and after on two lanes
    sim.set_controllers(0, [move_ctl("tangent_rotation", amp_move=0.3, amp_bead=amp, num_per_cycle=23, simple=False),
                            move_ctl("crank_shaft", amp_move=0.3, amp_bead=min(n, 9), num_per_cycle=11, simple=False)])
    sim.deposit(-1)
    sim.run(8, 5)
    sim.sync()
    out = sim.get_chain(0) + (sim.tally(0), np.array([c.acc_rate for c in sim.get_controllers(0)]), sim.energies()[0])
    sim.close()
    return out


@pytest.mark.parametrize("n,amp", [(2, 1), (2, 2), (9, 7), (9, 8), (10, 9), (17, 16), (40, 33), (300, 12), (300, 70)])
def test_four_lanes_a_bead(n, amp):
    want = _run(n, amp, 4, False)
    assert want[4][3, 1] > 0  # rotations were accepted
    for W in (1, 4, 12):
        for a, b in zip(want, _run(n, amp, W, True)):
            np.testing.assert_array_equal(a, b)
