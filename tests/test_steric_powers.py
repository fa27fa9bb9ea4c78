"""The clash energy of one pair against its exact value (rational arithmetic) for
the FP64 quotient f = e / d: f^12 - 2 f^6 + 1 within 2 units in the last place of
the terms' magnitudes.  Distances from just inside e to a thirtieth of it, and at 0,
where f^12 overflows and where it is not finite."""
from fractions import Fraction

import numpy as np
import pytest

from chromo_gb300 import _native as nat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fp64", [False, True])
def test_powers_are_correct_to_two_ulp(fp64):
    rng = np.random.default_rng(11)
    e = 10.0
    sim = nat.Sim([2], [[1, 1, 1]], 1, pos_fp64=fp64)
    sim.set_chain(0, r=np.array([[0.0, 0.0, 0.0], [1e3, 0.0, 0.0]]), t3=np.tile([1.0, 0, 0], (2, 1)),
                  t2=np.tile([0, 1.0, 0], (2, 1)))
    f = np.concatenate([rng.uniform(1.0, 1.3, 400), rng.uniform(1.3, 30.0, 400)])
    for x in e / f:
        got = sim.steric_delta(0, 1, 2, [[x, 0.0, 0.0]], e)  # from beyond e: the pair's energy
        q = Fraction(float(np.float64(e) / np.sqrt(np.float64(x) * np.float64(x))))
        want = q ** 12 - 2 * q ** 6 + 1 if x < e else Fraction(0)
        # 0.5 for each of the three sums and as much for the powers' own rounding
        assert abs(Fraction(got) - want) <= Fraction(2.0 ** -52) * 2 * (q ** 12 + 2 * q ** 6 + 1), x
    assert sim.steric_delta(0, 1, 2, [[1e-30, 0.0, 0.0]], e) == np.inf
    assert np.isnan(sim.steric_delta(0, 1, 2, [[0.0, 0.0, 0.0]], e))
    sim.close()
