"""Clash energies at the edges of the kernels' tiles (32 rows, 256 threads,
chunks of 1,024 columns), far from the origin, with pairs on both sides of the
excluded distance, against the oracle.

The device adds the same FP64 terms in another order: 1e-12 of the sum of the
terms' magnitudes (positions exact in the storage type)."""
import numpy as np
import pytest

from chromo_gb300 import _native as nat
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _chain(n, shift, seed):
    rng = np.random.default_rng(seed)
    r = np.cumsum(rng.normal(0.0, 4.0, (n, 3)), axis=0) * (60.0 / max(60.0, 4.0 * n ** 0.5)) + shift
    return r.astype(np.float32).astype(np.float64)


@pytest.mark.parametrize("fp64", [False, True])
@pytest.mark.parametrize("n", [2, 31, 33, 257, 1024, 1025, 2300])
@pytest.mark.parametrize("shift,e", [(0.0, 10.0), (9e4, 10.0), (0.0, 1e4)])
def test_steric_tiles_match_oracle(n, shift, e, fp64):
    r = _chain(n, shift, n)
    sim = nat.Sim([n], [[1, 1, 1]], 1, pos_fp64=fp64)
    sim.set_chain(0, r=r, t3=np.tile([1.0, 0, 0], (n, 1)), t2=np.tile([0, 1.0, 0], (n, 1)))
    want = orc.steric_energy(r, e)
    d = np.linalg.norm(r[:, None] - r[None], axis=2)[np.triu_indices(n, 1)]
    f6 = (e / d[d < e]) ** 6
    scale = float((f6 * f6 + 2 * f6 + 1).sum())
    assert abs(sim.steric_energy(0, e) - want) <= 1e-12 * scale + 1e-9
    rng = np.random.default_rng(n + 1)
    for ind0, indf in {(0, 1), (n - 1, n), (0, min(n, 33)), (max(0, n - 40), n), (n // 2, n // 2 + 1)}:
        trial = r[ind0:indf] + rng.normal(0.0, 3.0, (indf - ind0, 3))
        got, exp = sim.steric_delta(0, ind0, indf, trial, e), orc.steric_delta(r, trial, ind0, indf, e)
        moved = r.copy()
        moved[ind0:indf] = trial
        s = 0.0
        for x in (r, moved):
            dd = np.linalg.norm(x[ind0:indf, None] - x[None], axis=2)
            dd = dd[(dd < e) & (dd > 0)]
            g6 = (e / dd) ** 6
            s += float((g6 * g6 + 2 * g6 + 1).sum())
        assert abs(got - exp) <= 1e-12 * s + 1e-9, (ind0, indf, got, exp)
    sim.close()
