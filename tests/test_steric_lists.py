"""Clash energies where a thread of a tile takes four columns (chains and segments
of enough rows) and where a tile's list of near pairs is empty, part filled or too
short, against the oracle; tolerance as in test_steric_tiles.py.  Equal sums from
two calls: the list's order does not depend on timing."""
import numpy as np
import pytest

from chromo_gb300 import _native as nat
from oracle import oracle as orc
from test_steric_tiles import _chain

pytestmark = pytest.mark.gpu


def _terms(r, rows, e):
    d = np.linalg.norm(r[rows, None] - r[None], axis=2)
    d = d[(d < e) & (d > 0)]
    f6 = (e / d) ** 6
    return float((f6 * f6 + 2 * f6 + 1).sum())


@pytest.mark.parametrize("fp64", [False, True])
@pytest.mark.parametrize("n", [4100])
@pytest.mark.parametrize("e", [1e-3, 12.0, 25.0, 1e3])
def test_lists_match_oracle(n, e, fp64):
    r = _chain(n, 0.0, n)
    sim = nat.Sim([n], [[1, 1, 1]], 1, pos_fp64=fp64)
    sim.set_chain(0, r=r, t3=np.tile([1.0, 0, 0], (n, 1)), t2=np.tile([0, 1.0, 0], (n, 1)))
    got = sim.steric_energy(0, e)
    assert got == sim.steric_energy(0, e)
    assert abs(got - orc.steric_energy(r, e)) <= 1e-12 * _terms(r, np.arange(n), e) + 1e-9
    rng = np.random.default_rng(n)
    for ind0, indf in ((5, n - 7), (100, 101), (n - 70, n - 3)):
        trial = r[ind0:indf] + rng.normal(0.0, 3.0, (indf - ind0, 3))
        moved = r.copy()
        moved[ind0:indf] = trial
        rows = np.arange(ind0, indf)
        s = _terms(r, rows, e) + _terms(moved, rows, e)
        got = sim.steric_delta(0, ind0, indf, trial, e)
        assert got == sim.steric_delta(0, ind0, indf, trial, e)
        assert abs(got - orc.steric_delta(r, trial, ind0, indf, e)) <= 1e-12 * s + 1e-9, (ind0, indf)
    sim.close()
