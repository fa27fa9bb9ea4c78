"""fast_field with FP64 storage on the production kernel (a bead's axes on lanes, sub-bin
weights), move by move against the oracle's FP64 replay; bounds as for the FP64
configuration in test_gpu_spec_oracle.py (sin / cos differ in the last bit)."""
import numpy as np
import pytest

from golden_cases import gpu_sim, load, oracle_ctls, oracle_system
from test_gpu_spec_oracle import compare_records

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W", [0, 1, 5])
def test_fast_field_matches_oracle(W):
    g = load("fast_field")
    assert int(g["fast_n"]) > 0
    sim = gpu_sim(g, pos_fp64=True, warps_per_block=W)
    o = oracle_system(g, pos="f64", fixed_density=1)
    o.deposit_all()
    steps = 40
    cap = steps * int(sum(int(row[2]) for row in g["ctl0"])) + 10
    log = sim.run_logged(steps, 77, cap)[0]
    orecs, _, _ = o.mc_sim_philox(oracle_ctls(g), steps, 77, 0, 0, follow=log["accepted"])
    assert np.bincount(log["kind"][log["accepted"] == 1], minlength=5).min() > 0
    compare_records(log, orecs, tol=1e-9, label="fast_field fp64")
    r, t3, t2, st = sim.get_chain(0)
    for a, b in ((r, o.r), (t3, o.t3), (t2, o.t2)):
        np.testing.assert_allclose(a, b, rtol=1e-9, atol=1e-9)
    np.testing.assert_array_equal(st, o.states)
    assert np.abs(sim.density(0) - o.density_fx).max() <= 16
    sim.close()
