"""Default launch shapes of many replicas: each leaves room for a pooled voxel table
(fewer warps, then fewer CTAs per SM, than would otherwise run), whose state equals
one move at a time bit for bit."""
import numpy as np
import pytest

from chromo_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fp64", [False, True])
@pytest.mark.parametrize("R,nb", [(1064, 2), (1216, 1), (1216, 3), (1672, 2), (2433, 2), (2433, 3)])
def test_default_shape_has_a_pooled_table(R, nb, fp64):
    rng = np.random.default_rng(R)
    w = wl.Workload("many", np.full(R, 40), 7, nb, rng.uniform(-1, 0, size=(R, nb)), np.ones(R), [-4.0, -3.0, -2.0][:nb],
                    [{}] * nb, 20, 0, wl.BASE_SEED + R)
    chains = wl.make_chains(w)
    out = []
    for W in (0, 1):
        sim = wl.build_sim(w, chains, pos_fp64=fp64, warps_per_block=W)
        if W == 0:
            assert sim.launch_shape()[3] >= 256  # a slot's own table would have at most 128 entries here
        sim.run(1, 3)
        sim.sync()
        out.append([sim.get_chain(r) + (sim.tally(r),) for r in range(0, R, 97)])
        sim.close()
    for a, b in zip(*out):
        for x, y in zip(a, b):
            np.testing.assert_array_equal(x, y)
