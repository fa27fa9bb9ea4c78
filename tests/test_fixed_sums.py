"""Sums of products of the grid's fixed-point columns at the edges of their integer
form: columns just below and above 2^52 (4,096 beads' weight in one voxel), above
vf_limit and not, and more voxels than a thread's 64-bit sums hold, against the
NumPy restatement and tolerance of test_sums.py."""
import numpy as np
import pytest

from test_sums import _case, _field

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dims,nb,kw", [
    (2040, (1, 1, 1), 2, dict(vf_limit=1e6)),   # below 2^52, states' columns too
    (4096, (1, 1, 1), 3, dict(vf_limit=1e6)),   # at it
    (6000, (1, 1, 2), 3, dict(vf_limit=1e6)),   # some columns of a row above it
    (6000, (1, 1, 1), 2, dict(vf_limit=0.5)),   # above it and above vf_limit
    (500, (165, 165, 165), 3, {}),              # 2,194 rows a thread
    (300, (260, 261, 262), 1, {})])             # 8,681 rows a thread
def test_column_sums(n, dims, nb, kw):
    sim, c, bonds, p = _case(n, dims, nb, n, **kw)
    e = sim.energies()[0]
    _, T = sim.gradient(False, True)
    T = T[0]
    sim.close()
    want_fe, S, rho, dens = _field(c["r"], c["states"], p)
    scale = abs(p["chi"] * S) + sum(abs(p["pref"][b]) * (rho[b] ** 2).sum() for b in range(nb)) + n
    np.testing.assert_allclose(e[2], want_fe, rtol=1e-9, atol=1e-9 * scale)
    np.testing.assert_allclose(e[4], S, rtol=1e-9, atol=1e-12)
    want = [S] + [(rho[b] ** 2).sum() if b < nb else 0.0 for b in range(3)]
    want += [(rho[b] * rho[q]).sum() if q < nb else 0.0 for b, q in ((0, 1), (0, 2), (1, 2))]
    np.testing.assert_allclose(T[:7], want, rtol=1e-9, atol=1e-13)
    np.testing.assert_allclose(T[13], (dens ** 2).sum(), rtol=1e-9)
