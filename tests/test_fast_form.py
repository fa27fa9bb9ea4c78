"""fast_field replicas in the MC kernel's form for them (no SSTWLC or move-log code) against
the full form, which a logged run takes: the same bits, for each storage and number of
lanes, with every replica or only some in fast_field."""
import numpy as np
import pytest

from chromo_gb300 import workloads as wl
from chromo_gb300.device import field_params
from golden_cases import gpu_sim, load

pytestmark = pytest.mark.gpu
CAP = 100000


@pytest.mark.parametrize("fp64,G,W", [(False, 32, 0), (False, 16, 0), (False, 8, 2), (True, 32, 0), (False, 32, 1)])
def test_form_with_sub_bins_equals_full_form(fp64, G, W):
    g = load("fast_field")
    assert int(g["fast_n"]) > 0
    out = []
    for logged in (False, True):
        sim = gpu_sim(g, pos_fp64=fp64, warps_per_block=W, lanes_per_move=G)
        if logged:
            sim.run_logged(30, 5, CAP)
        else:
            sim.run(30, 5)
        sim.sync()
        out.append(sim.get_chain(0) + (sim.tally(0), sim.density(0), sim.energies()))
        sim.close()
    assert out[0][4][:, 1].sum() > 0
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


def test_captured_rounds_take_the_form_of_the_fields():
    """Rounds captured without fast_field, then with it on one of two replicas of equal chi:
    the chains of one move at a time in the full form."""
    w = wl.Workload("form", np.array([300, 260]), 7, 1, np.zeros((2, 1)), np.ones(2), [-4.0], [{}], 20, 0, 3)
    chains = wl.make_chains(w)
    fast = field_params(field_kind=2, nxyz=(7,) * 3, widths=(7 * wl.VOXEL,) * 3, n_binders=1, chi=1.0, vf_limit=0.5,
                        bead_vol=4.0 / 3.0 * np.pi * wl.BEAD_RAD ** 3, pref=[-2e5], intra=[-1.0], fast_field=1, n_points=64)
    out = []
    for rounds in (True, False):
        sim = wl.build_sim(w, chains, warps_per_block=0 if rounds else 1)
        for k in range(2):
            if k:
                sim.set_field(1, fast)
            if rounds:
                sim.run_batched(2, 3, 2, 9)
            else:
                sim.run_logged(6, 9, CAP)
            sim.sync()
        out.append([x for r in range(2) for x in sim.get_chain(r) + (sim.density(r),)])
        sim.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
