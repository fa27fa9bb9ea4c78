"""The library's default launch shapes (more warps than moves in flight, moves in
flight chosen from the conflicts met) against one move at a time: one CTA per
SM, two and three, on chains short enough that most batches are cut."""
import numpy as np
import pytest

from chromo_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R,n", [(1, 400), (160, 160), (310, 200)])
def test_default_shape_equals_sequential(R, n):
    rng = np.random.default_rng(R)
    w = wl.Workload("shape", np.full(R, n), 7, 2, rng.uniform(-1, 0, size=(R, 2)), np.ones(R), [-4.0, -3.0],
                    [{"PRC1": 1.0}, {}], 20, 0, wl.BASE_SEED + R)
    chains = wl.make_chains(w)
    out = []
    for W in (0, 1):
        sim = wl.build_sim(w, chains, warps_per_block=W)
        if W == 0:
            warps, lanes, moves, _ = sim.launch_shape()
            assert lanes == 32 and (moves < warps or warps <= 3)
        sim.run(6, 3)
        sim.sync()
        out.append([sim.get_chain(r) + (sim.tally(r), np.array([c.acc_rate for c in sim.get_controllers(r)]))
                    for r in range(R)] + [sim.energies()])
        sim.close()
    for a, b in zip(out[0][:-1], out[1][:-1]):
        for x, y in zip(a, b):
            np.testing.assert_array_equal(x, y)
    np.testing.assert_array_equal(out[0][-1], out[1][-1])
