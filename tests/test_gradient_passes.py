"""dE/dr where the kernel takes several passes a warp, and where a coordinate's
cells come from the general remainder: the same values bit for bit as one pass a
warp and as the coordinates inside 2^20 boxes."""
import numpy as np
import pytest

from chromo_gb300 import _native as nat
from chromo_gb300.device import bonds_array, field_params
from chromo_gb300.energetics import dss_parameters

pytestmark = pytest.mark.gpu
W = 256.0  # box width: multiples of it are exact in FP64


def _sim(R, n, r, fp64):
    rng = np.random.default_rng(n)
    t3 = rng.normal(size=(n, 3))
    t3 /= np.linalg.norm(t3, axis=1)[:, None]
    states = rng.integers(0, 3, size=(n, 2))
    _, eb, g, ep, epp, eta = dss_parameters(np.full(n - 1, 16.5), 53.0)
    sim = nat.Sim([n] * R, [(8, 8, 8)] * R, 2, pos_fp64=fp64)
    for k in range(R):
        sim.set_chain(k, r=r, t3=t3, t2=np.roll(t3, 1, axis=1), states=states, marks=np.zeros((n, 2), np.int64),
                      bonds=bonds_array(eb, g, ep, epp, eta))
        sim.set_field(k, field_params(field_kind=2, nxyz=(8, 8, 8), widths=(W,) * 3, n_binders=2, chi=1.3,
                                      vf_limit=1e6, bead_vol=523.6, pref=[-900.0, 400.0], intra=[-4.0, 0.0]))
    sim.deposit(-1)
    return sim


def _walk(n):
    rng = np.random.default_rng(5)
    return np.round(np.cumsum(rng.normal(size=(n, 3)) * 10.0, axis=0) * 2.0 ** 10) / 2.0 ** 10


@pytest.mark.parametrize("fp64", [False, True])
@pytest.mark.parametrize("R,n", [(40, 7000), (100, 3041), (3, 250000)])
def test_passes_agree(R, n, fp64):
    r = _walk(n)
    one = _sim(1, n, r, fp64)
    want, _ = one.gradient(True, False)
    one.close()
    sim = _sim(R, n, r, fp64)
    got, _ = sim.gradient(True, False)
    sim.close()
    got = np.asarray(got).reshape(R, n, 3)
    for k in range(R):
        np.testing.assert_array_equal(got[k], np.asarray(want).reshape(n, 3))


@pytest.mark.parametrize("boxes", [1.0, -3.0, 2.0 ** 21, -(2.0 ** 22)])
def test_far_coordinates(boxes):
    n = 500
    r = _walk(n)
    out = []
    for shift in (0.0, boxes * W):
        sim = _sim(1, n, r + shift, True)
        out.append(np.asarray(sim.gradient(True, False)[0]))
        sim.close()
    np.testing.assert_array_equal(out[0], out[1])
