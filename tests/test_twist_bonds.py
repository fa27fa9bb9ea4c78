"""Twist energies of the boundary bonds of an SSTWLC chain's position moves: one
energy per lane, packed over the last warps of the CTA, or after the beads where
these warps would be more than half of it.  The state after a run does not depend
on the launch shape, and for FP64 storage the sum of the accepted changes is the
recomputed energy's change up to rounding."""
import numpy as np
import pytest

from chromo_gb300 import _native as nat
from chromo_gb300 import synthetic as syn
from chromo_gb300.device import binding_params, bonds_array, field_params, move_ctl
from chromo_gb300.energetics import dss_parameters

pytestmark = pytest.mark.gpu


def _run(n, amp, W, G, fp64):
    rng = np.random.default_rng(n)
    r = syn.gaussian_walk(rng, n, 16.5)
    t3, t2 = syn.tangents_from_coordinates(r)
    _, eb, g, ep, epp, eta = dss_parameters(np.full(n - 1, 16.5), 53.0)
    sim = nat.Sim([n], [(6, 6, 6)], 1, pos_fp64=fp64, max_segment=amp + 2, max_tangent=n, warps_per_block=W,
                  lanes_per_move=G)
    sim.set_chain(0, r=r, t3=t3, t2=t2, states=np.zeros((n, 1), np.int64), marks=np.zeros((n, 1), np.int64),
                  bonds=bonds_array(eb, g, ep, epp, eta))
    sim.set_twist(0, np.full(n - 1, 6.0), np.full(n - 1, 16.5 * 2 * np.pi / 10.5 / 0.332))
    sim.set_field(0, field_params(field_kind=2, nxyz=(6, 6, 6), widths=(240.0,) * 3, n_binders=1, bead_vol=523.6,
                                  pref=[0.0], intra=[0.0]))
    sim.set_binding(0, binding_params(sites=[2], e_mod=[0.0], e_nomod=[0.0], mu=[0.0]))
    sim.set_controllers(0, [move_ctl(m, amp_move=0.3 if m != "slide" else 2.0, amp_bead=amp, num_per_cycle=37,
                                     simple=False) for m in ("crank_shaft", "end_pivot", "slide")])
    sim.deposit(-1)
    before = sim.energies()[0]
    sim.run(6, 5)
    sim.sync()
    after = sim.energies()[0]
    out = sim.get_chain(0) + (sim.tally(0),)
    sim.close()
    return out, before, after


@pytest.mark.parametrize("fp64", [False, True])
@pytest.mark.parametrize("n,amp", [(2, 1), (5, 3), (40, 12), (2000, 30)])
def test_any_launch_shape_and_exact_sum(n, amp, fp64):
    want, before, after = _run(n, amp, 1, 32, fp64)
    assert want[-1][:3, 1].sum() > 0  # moves were accepted
    if fp64:
        # ~200 moves whose terms reach ~1e2 kT, FP64 rounding 1e-16 each
        assert abs((after[:3] - before[:3]).sum() - (after[3] - before[3])) <= 1e-9 * max(1.0, abs(before[:3]).sum())
    for W, G in ((2, 32), (5, 32), (12, 32)) + (() if fp64 else ((1, 8), (3, 8))):
        for a, b in zip(want, _run(n, amp, W, G, fp64)[0]):
            np.testing.assert_array_equal(a, b)
