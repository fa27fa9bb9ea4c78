"""Position moves at the edges of the CTA's pooled voxel table: many long
segments in flight (the pool overflows; segments over 256 beads never enter it),
a grid of 2^26 voxels (no pool: each slot's own table) and grids with axes of a
single voxel (a bead's corners share it, the most that an entry's split counters
hold).  Several moves in flight equal one at a time bit for bit, and the grid
equals its re-deposit."""
import numpy as np
import pytest

from chromo_gb300 import _native as nat
from chromo_gb300 import synthetic as syn
from chromo_gb300.device import binding_params, bonds_array, field_params, move_ctl
from chromo_gb300.energetics import dss_parameters

pytestmark = pytest.mark.gpu


def _sim(n, dims, amp, fp64, W):
    rng = np.random.default_rng(17)
    r = syn.gaussian_walk(rng, n, 16.5)
    t3, t2 = syn.tangents_from_coordinates(r)
    marks = syn.markov_marks(rng, n, 20)[:, None]
    states = rng.integers(0, 3, size=(n, 1))
    _, eb, g, ep, epp, eta = dss_parameters(np.full(n - 1, 16.5), 53.0)
    sim = nat.Sim([n], [dims], 1, pos_fp64=fp64, max_segment=amp + 2, max_tangent=n, warps_per_block=W)
    sim.set_chain(0, r=r, t3=t3, t2=t2, states=states, marks=marks, bonds=bonds_array(eb, g, ep, epp, eta))
    sim.set_field(0, field_params(field_kind=2, nxyz=dims, widths=tuple(40.0 * d for d in dims), n_binders=1,
                                  chi=1.0, vf_limit=1e6, bead_vol=523.6, pref=[-100.0], intra=[-3.9]))
    sim.set_binding(0, binding_params(sites=[2], e_mod=[-0.01], e_nomod=[1.52], mu=[-0.4]))
    sim.set_controllers(0, [move_ctl(m, amp_move=0.2 if m != "slide" else 2.0, amp_bead=amp, num_per_cycle=24,
                                     simple=False) for m in ("crank_shaft", "end_pivot", "slide")])
    sim.deposit(-1)
    return sim


@pytest.mark.parametrize("fp64", [False, True])
@pytest.mark.parametrize("n,dims,amp", [(3000, (20, 21, 22), 600), (400, (30, 30, 30), 255), (500, (8192, 8192, 1), 120),
                                        (400, (1, 1, 1), 255), (400, (1, 40, 1), 200)])
def test_long_moves_and_large_grids_equal_sequential(n, dims, amp, fp64):
    got = []
    for W in (1, 12):
        sim = _sim(n, dims, amp, fp64, W)
        sim.run(2, 99)
        sim.sync()
        field, small = sim.energy(0)[2], np.prod(dims) < 1e6
        grid = sim.density(0) if small else None
        chain = sim.get_chain(0)
        sim.deposit(-1)
        np.testing.assert_allclose(sim.energy(0)[2], field, rtol=1e-12)
        if small:
            np.testing.assert_array_equal(sim.density(0), grid)
        got.append(chain + (sim.tally(0),))
        sim.close()
    assert got[0][-1][:3, 1].sum() > 0  # moves were accepted
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)
