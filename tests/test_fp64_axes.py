"""FP64 storage: a bead's three axes on three lanes, the remainder, the quotient
by the voxel width and the field's quotients in integer steps and FMAs -- moves of
one bead to many, boxes of one voxel, odd ones, tiny and huge ones (where the
general division and remainder are taken), coordinates beyond 2^20 boxes, with and
without confinement.  After a run the grid is the deposit of the beads bit for
bit, the state does not depend on the number of warps, and the sum of the accepted
changes is the recomputed energy's change up to rounding."""
import numpy as np
import pytest

from chromo_gb300 import _native as nat
from chromo_gb300 import synthetic as syn
from chromo_gb300.device import binding_params, bonds_array, field_params, move_ctl
from chromo_gb300.energetics import dss_parameters

pytestmark = pytest.mark.gpu


def _run(n, dims, voxel, amp, shift, confine, W):
    rng = np.random.default_rng(n)
    r = syn.gaussian_walk(rng, n, 16.5) + shift
    t3, t2 = syn.tangents_from_coordinates(r - shift)
    marks = syn.markov_marks(rng, n, 20)[:, None]
    _, eb, g, ep, epp, eta = dss_parameters(np.full(n - 1, 16.5), 53.0)
    sim = nat.Sim([n], [dims], 1, pos_fp64=True, max_segment=amp + 2, max_tangent=n, warps_per_block=W)
    sim.set_chain(0, r=r, t3=t3, t2=t2, states=rng.integers(0, 3, size=(n, 1)), marks=marks,
                  bonds=bonds_array(eb, g, ep, epp, eta))
    sim.set_field(0, field_params(field_kind=2, nxyz=dims, widths=tuple(voxel * d for d in dims), n_binders=1,
                                  chi=1.0, vf_limit=1e300, bead_vol=523.6 * (voxel / 40.0) ** 3,
                                  pref=[-100.0 * voxel ** 3], intra=[-3.9], confine_kind=confine,
                                  confine_length=900.0))
    sim.set_binding(0, binding_params(sites=[2], e_mod=[-0.01], e_nomod=[1.52], mu=[-0.4]))
    sim.set_controllers(0, [move_ctl(m, amp_move=0.2 if m != "slide" else 2.0, amp_bead=amp, num_per_cycle=13,
                                     simple=False) for m in ("crank_shaft", "end_pivot", "slide")])
    sim.deposit(-1)
    before = sim.energies()[0]
    sim.run(4, 9)
    sim.sync()
    after, grid = sim.energies()[0], sim.density(0)
    out = sim.get_chain(0) + (sim.tally(0),)
    sim.deposit(-1)
    np.testing.assert_array_equal(sim.density(0), grid)
    sim.close()
    return out, before, after


@pytest.mark.parametrize("n,dims,voxel,amp,shift,confine", [
    (2, (3, 4, 5), 40.0, 1, 0.0, 0), (9, (1, 1, 1), 40.0, 7, 0.0, 1), (33, (7, 1, 3), 33.3, 8, 0.0, 2),
    (300, (30, 29, 31), 40.0, 120, 0.0, 1), (300, (8, 8, 8), 1.0 / 3.0, 33, 0.0, 0),
    (120, (5, 6, 7), 40.0, 30, 3e9, 0),          # beyond 2^20 boxes
    (60, (4, 4, 4), 1e-36, 20, 0.0, 0),          # a box and a volume below the integer steps' range
    (60, (4, 4, 4), 1e40, 20, 0.0, 0)])          # and above it
def test_any_box_and_warps(n, dims, voxel, amp, shift, confine):
    want, before, after = _run(n, dims, voxel, amp, shift, confine, 1)
    if shift == 0.0 and voxel > 1e-3:
        assert want[-1][:3, 1].sum() > 0  # moves were accepted
        # ~100 moves, terms up to the energies' size, FP64 rounding; the grid's
        # fixed point (2^-41 a weight) leaves ~1e-12 of the field
        size = max(1.0, np.abs(before[:3]).sum(), np.abs(after[:3]).sum())
        assert abs((after[:3] - before[:3]).sum() - (after[3] - before[3])) <= 1e-9 * size
    for W in (2, 12):
        for a, b in zip(want, _run(n, dims, voxel, amp, shift, confine, W)[0]):
            np.testing.assert_array_equal(a, b)
