"""The clash energy of one pair, f^12 - 2 f^6 + 1 with f = e / d, against its exact value
(rational arithmetic): no further from it, in root mean square over the terms'
magnitudes, than pow(e / d, 12) and pow(e / d, 6) in FP64.  Distances from just inside
e to a thirtieth of it; distances where f^12 overflows and where it is not finite; and
excluded distances whose squares leave FP64's range."""
from fractions import Fraction

import numpy as np
import pytest

from chromo_gb300 import _native as nat

pytestmark = pytest.mark.gpu


def _pair(fp64):
    sim = nat.Sim([2], [[1, 1, 1]], 1, pos_fp64=fp64)
    sim.set_chain(0, r=np.array([[0.0, 0.0, 0.0], [1e3, 0.0, 0.0]]), t3=np.tile([1.0, 0, 0], (2, 1)),
                  t2=np.tile([0, 1.0, 0], (2, 1)))
    return sim


@pytest.mark.parametrize("fp64", [False, True])
@pytest.mark.parametrize("low,high", [(1.0, 1.3), (1.0, 3.0), (1.3, 30.0)])
def test_no_further_from_exact_than_pow(low, high, fp64):
    rng = np.random.default_rng(11)
    e = 10.0
    sim = _pair(fp64)
    got, ref = [], []
    for x in (e / rng.uniform(low, high, 400))[:, None] * np.array([0.6, 0.64, 0.48]):
        q = Fraction(e) ** 2 / sum(Fraction(float(v)) ** 2 for v in x)
        if q <= 1:
            continue
        want, size = q ** 6 - 2 * q ** 3 + 1, q ** 6 + 2 * q ** 3 + 1
        f = e / np.sqrt(x[0] * x[0] + x[1] * x[1] + x[2] * x[2])
        # from beyond e: the change is the pair's energy
        got.append(float((Fraction(sim.steric_delta(0, 1, 2, [x], e)) - want) / size))
        ref.append(float((Fraction(float(f ** 12.0 - 2 * f ** 6.0 + 1)) - want) / size))
    sim.close()
    assert len(got) > 300
    assert np.sqrt(np.mean(np.square(got))) <= np.sqrt(np.mean(np.square(ref)))


@pytest.mark.parametrize("fp64", [False, True])
def test_ends_of_the_range(fp64):
    sim = _pair(fp64)
    assert sim.steric_delta(0, 1, 2, [[1e-30, 0.0, 0.0]], 10.0) == np.inf
    assert np.isnan(sim.steric_delta(0, 1, 2, [[0.0, 0.0, 0.0]], 10.0))
    assert sim.steric_delta(0, 1, 2, [[10.0, 0.0, 0.0]], 10.0) == 0.0
    # e^2 out of range: bead 1 from f = 2 to f = 4 at a huge distance, from beyond e at a tiny one
    for scale in (2.0 ** 600, 2.0 ** -510):
        big = nat.Sim([2], [[1, 1, 1]], 1, pos_fp64=True)
        start = 0.5 if scale > 1 else 2.0
        big.set_chain(0, r=np.array([[0.0, 0.0, 0.0], [start * scale, 0.0, 0.0]]))
        change = big.steric_delta(0, 1, 2, [[0.25 * scale, 0.0, 0.0]], scale)
        f6 = np.array([4.0, 2.0]) ** 6
        e = f6 * f6 - 2 * f6 + 1
        assert change == (0.0 if scale > 1 else e[0])  # beyond 2^512 the squared distance is infinite: no clash
        big.close()
    sim.close()
