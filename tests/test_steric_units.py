"""Clash energies do not depend on the unit of length: a chain and an excluded
distance scaled by a power of two (exact in both storage types) give the unscaled
chain's energy and change, also where squared distances leave FP32's range.  The
same terms in another order: 1e-12 of their magnitudes."""
import numpy as np
import pytest

from chromo_gb300 import _native as nat
from test_steric_tiles import _chain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fp64,power", [(False, -60), (False, -80), (False, -110), (False, 80), (True, -64), (True, -160),
                                        (True, 160)])
@pytest.mark.parametrize("n", [70, 1100])
def test_any_unit_of_length(n, power, fp64):
    r, e = _chain(n, 0.0, n), 12.0
    rng = np.random.default_rng(n)
    ind0, indf = 20, 61
    trial = r[ind0:indf] + rng.normal(0.0, 3.0, (indf - ind0, 3))
    f6 = (e / np.linalg.norm(np.concatenate([r, trial])[:, None] - np.concatenate([r, trial])[None], axis=2)[
        np.triu_indices(n + len(trial), 1)]) ** 6
    f6 = f6[(f6 > 1) & np.isfinite(f6)]
    size = float((f6 * f6 + 2 * f6 + 1).sum())
    got = []
    for s in (1.0, 2.0 ** power):
        sim = nat.Sim([n], [[1, 1, 1]], 1, pos_fp64=fp64)
        sim.set_chain(0, r=r * s, t3=np.tile([1.0, 0, 0], (n, 1)), t2=np.tile([0, 1.0, 0], (n, 1)))
        got.append((sim.steric_energy(0, e * s), sim.steric_delta(0, ind0, indf, trial * s, e * s)))
        sim.close()
    assert got[0][0] > 0.0 and got[0][1] != 0.0
    for a, b in zip(*got):
        assert abs(a - b) <= 1e-12 * size
