"""Energies, exchange sums, derivative terms and dE/dr at the edges of the
kernels' tiles: chains of 2 beads to a few around the 30 and 31 beads a warp
takes per pass and the eighths of a cluster, one to three binders, grids with
odd and single-voxel axes, voxels above vf_limit, a binding cap and a confining
sphere's volumes, against a NumPy restatement.

FP64 storage: the grid's fixed point rounds each weight to 2^-41, so sums over
voxels agree to ~1e-11 relative; 1e-9 is asked."""
import numpy as np
import pytest

from chromo_gb300 import _native as nat
from chromo_gb300.device import binding_params, bonds_array, field_params
from chromo_gb300.energetics import binding_free_energy_table, dss_parameters
from energy_model import binding, elastic, trilinear, voxel_fraction

pytestmark = pytest.mark.gpu
BEAD_VOL, D = 523.6, 40.0


def _case(n, dims, nb, seed, vf_limit=0.5, cap=-1, access=False, fp64=True):
    rng = np.random.default_rng(seed)
    step = rng.normal(size=(n, 3))
    t3 = step / np.linalg.norm(step, axis=1)[:, None]
    r = np.cumsum(10.0 * step, axis=0).astype(np.float32).astype(np.float64)
    t3 = t3.astype(np.float32).astype(np.float64)
    c = dict(r=r, t3=t3, t2=np.roll(t3, 1, axis=1), states=rng.integers(0, 3, size=(n, nb)),
             marks=rng.integers(0, 3, size=(n, nb)))
    _, eb, g, ep, epp, eta = dss_parameters(np.full(n - 1, 16.5), 53.0)
    bonds = bonds_array(eb, g, ep, epp, eta)
    xpref = np.zeros((nb, nb))
    if nb > 1:
        xpref[0, 1], xpref[1, nb - 1] = 900.0, -700.0
    V = np.full(int(np.prod(dims)), D ** 3)
    if access:
        V = V * rng.uniform(0.2, 1.0, V.size)
    p = dict(widths=[D * d for d in dims], n=list(dims), V=V, chi=1.3, vf_limit=vf_limit, cap=cap,
             pref=[-900.0 - 100 * b for b in range(nb)], intra=[-4.0 + b for b in range(nb)], xpref=xpref,
             mu=[-0.4, 0.3, -0.1][:nb], adj=0.9)
    p["bind_f"] = np.asarray(binding_free_energy_table([2] * nb, [-0.01] * nb, [1.52] * nb))
    sim = nat.Sim([n], [dims], nb, pos_fp64=fp64, nonuniform_access=access)
    sim.set_chain(0, bonds=bonds, **c)
    sim.set_field(0, field_params(field_kind=2, nxyz=dims, widths=tuple(p["widths"]), n_binders=nb, chi=p["chi"],
                                  vf_limit=vf_limit, bead_vol=BEAD_VOL, pref=p["pref"], intra=p["intra"],
                                  xpref=xpref), access_vol=V if access else None)
    sim.set_binding(0, binding_params(sites=[2] * nb, e_mod=[-0.01] * nb, e_nomod=[1.52] * nb, mu=p["mu"],
                                      mu_adjust_factor=p["adj"], max_binders=cap))
    sim.deposit(-1)
    return sim, c, bonds, p


def _grid(r, states, p):
    idx, w = trilinear(r, p["widths"], p["n"])
    cols = [np.ones(len(r))] + list(states.T.astype(float))
    out = np.zeros((len(cols), len(p["V"])))
    for k, s in enumerate(cols):
        np.add.at(out[k], idx.ravel(), (w * s[:, None]).ravel())
    return out


def _field(r, states, p):
    g = _grid(r, states, p) / p["V"]
    rho, vf = g[1:], g[0] * BEAD_VOL
    over = vf > p["vf_limit"]
    sv = np.where(over, 0.0, p["V"] / BEAD_VOL * vf * vf)
    e = p["chi"] * sv.sum() + 1e99 * vf[over].sum()
    for b in range(len(rho)):
        e += p["pref"][b] * (rho[b] ** 2).sum() + p["intra"][b] * (states[:, b] == 2).sum()
        for k in range(len(rho)):
            e += p["xpref"][b, k] * (rho[b] * rho[k]).sum()
    return e, sv.sum(), rho, g[0]


@pytest.mark.parametrize("n,dims,nb,kw", [
    (2, (5, 5, 5), 1, {}), (7, (1, 3, 1), 2, {}), (30, (4, 5, 6), 2, {}), (31, (7, 3, 5), 3, {}),
    (32, (9, 9, 9), 1, {}), (33, (2, 2, 2), 2, {}), (62, (8, 1, 9), 3, {}), (249, (11, 10, 9), 2, {}),
    (1985, (33, 31, 7), 3, {}), (400, (3, 4, 3), 2, dict(vf_limit=0.05)), (300, (6, 6, 6), 2, dict(cap=1)),
    (300, (13, 12, 11), 2, dict(access=True)), (200, (4, 4, 4), 3, dict(access=True, vf_limit=0.03)),
    (120, (5, 5, 5), 2, dict(vf_limit=0.0)), (120, (5, 5, 5), 1, dict(vf_limit=-1.0))])
def test_sums_match_restatement(n, dims, nb, kw):
    sim, c, bonds, p = _case(n, dims, nb, n, **kw)
    e = sim.energies()[0]
    _, T = sim.gradient()
    T = T[0]
    sim.close()
    want_fe, S, rho, dens = _field(c["r"], c["states"], p)
    tot = c["states"].sum(axis=1)
    want_bi = binding(c["states"], c["marks"], p)
    if p["cap"] >= 0:
        want_bi += 1e25 * np.maximum(0, tot - p["cap"]).sum()
    np.testing.assert_allclose(e[0], elastic(c["r"], c["t3"], bonds), rtol=1e-12)
    np.testing.assert_allclose(e[1], want_bi, rtol=1e-12)
    scale = abs(p["chi"] * S) + sum(abs(p["pref"][b]) * (rho[b] ** 2).sum() for b in range(nb)) + n
    np.testing.assert_allclose(e[2], want_fe, rtol=1e-9, atol=1e-9 * scale)
    np.testing.assert_allclose(e[4], S, rtol=1e-9, atol=1e-12)
    want = np.zeros(14)
    want[0], want[13] = S, (dens ** 2).sum()
    for b in range(nb):
        want[1 + b] = (rho[b] ** 2).sum()
        want[7 + b], want[10 + b] = (c["states"][:, b] == 2).sum(), c["states"][:, b].sum()
    for k, (b, q) in enumerate(((0, 1), (0, 2), (1, 2))):
        want[4 + k] = (rho[b] * rho[q]).sum() if q < nb else 0.0
    np.testing.assert_allclose(T, want, rtol=1e-9, atol=1e-13)


@pytest.mark.parametrize("n,dims,nb,access", [(2, (6, 5, 7), 1, False), (30, (6, 5, 7), 2, False),
                                              (31, (6, 5, 7), 3, False), (61, (9, 8, 2), 2, True),
                                              (121, (7, 7, 7), 2, False)])
@pytest.mark.parametrize("fp64", [False, True])
def test_gradient_matches_finite_differences(n, dims, nb, access, fp64):
    """Every bead's dE/dr against FP64 central differences (h = 1e-4; the
    energy's third derivatives leave ~1e-7 relative; coordinates within 1e-3 of
    a voxel face are skipped).  FP32 storage: the grid is deposited with FP32
    weights, good to ~1e-6 of a density; 1e-4 is asked of both."""
    sim, c, bonds, p = _case(n, dims, nb, 100 + n, access=access, fp64=fp64)
    g, _ = sim.gradient(True, False)
    sim.close()
    h = 1e-4
    frac = voxel_fraction(c["r"], p["widths"], p["n"])

    def E(r):
        return elastic(r, c["t3"], bonds) + _field(r, c["states"], p)[0]

    for i in sorted({0, 1, 2, n - 3, n - 2, n - 1, 28, 29, 30, 31, 32, 59, 60, 61, 119, 120} & set(range(n))):
        for j in range(3):
            if min(frac[i, j], 1 - frac[i, j]) < 1e-3:
                continue
            a, b = c["r"].copy(), c["r"].copy()
            a[i, j] += h
            b[i, j] -= h
            fd = (E(a) - E(b)) / (2 * h)
            assert abs(g[i, j] - fd) <= 1e-4 * max(1.0, abs(fd)), (i, j, g[i, j], fd)
