"""Deposits of beads far outside the periodic box, on its faces and at
multiples of its width: the grid equals the wrap of numpy's fmod bit for bit
(the FP64 remainder on the device takes fmod only for coordinates beyond 2^20
boxes)."""
import numpy as np
import pytest

from chromo_gb300 import _native as nat
from chromo_gb300.device import field_params

pytestmark = pytest.mark.gpu


def _coordinates(width, dtype):
    w = dtype(width)
    k = np.array([0, 1, 2, 3, 7, 1000, 2 ** 19, 2 ** 20 - 1, 2 ** 20, 2 ** 21], dtype=dtype)
    base = (k[:, None] * w + w * dtype(0.5) * np.array([-1, 0, 1], dtype=dtype)).ravel()
    near = np.concatenate([base, np.nextafter(base, dtype(np.inf)), np.nextafter(base, dtype(-np.inf)),
                           base + w * dtype(0.3), [dtype(1e-30), dtype(0.0)]]).astype(dtype)
    return np.concatenate([near, -near])


def _grid(r, n, width, dtype):
    """The fixed-point bead weights of positions r [N, 3] (arithmetic in dtype)."""
    w, half = dtype(width), dtype(0.5 * width)
    d64 = np.float64(width) / n
    y = (r + half).astype(dtype)
    m = np.fmod(y, w)
    m = np.where((m != 0) & (m < 0), (m + w).astype(dtype), m)
    x = np.where((y >= 0) & (y < w), y, m)
    x = (x - dtype(0.5 * d64)).astype(dtype)
    t = (x * dtype(1.0 / d64)).astype(dtype) if dtype is np.float32 else x / d64
    fl = np.floor(t)
    ind = fl.astype(np.int64)
    lo = np.clip(np.where(ind == -1, n - 1, ind), 0, n - 1)
    hi = np.where(lo + 1 == n, 0, lo + 1)
    wl = (dtype(1) - (t - fl).astype(dtype)).astype(dtype)
    g = np.zeros(n ** 3, dtype=np.int64)
    for c in range(8):
        bit = [(c >> j) & 1 for j in range(3)]
        f = [(dtype(1) - wl[:, j]).astype(dtype) if bit[j] else wl[:, j] for j in range(3)]
        wt = ((f[0] * f[1]).astype(dtype) * f[2]).astype(dtype)
        v = [hi[:, j] if bit[j] else lo[:, j] for j in range(3)]
        np.add.at(g, v[0] + n * (v[1] + n * v[2]), np.rint(wt.astype(np.float64) * 2.0 ** 40).astype(np.int64))
    return g


@pytest.mark.parametrize("fp64", [False, True])
@pytest.mark.parametrize("n,width", [(30, 1200.0), (7, 333.3), (1, 40.0)])
def test_deposit_wraps_as_fmod(fp64, n, width):
    dtype = np.float64 if fp64 else np.float32
    c = _coordinates(width, dtype)
    rng = np.random.default_rng(3)
    r = np.stack([rng.permutation(c) for _ in range(3)], axis=1)
    N = len(r)
    sim = nat.Sim([N], [[n] * 3], 1, pos_fp64=fp64)
    sim.set_chain(0, r=r, t3=np.tile([0.0, 0, 1], (N, 1)), t2=np.tile([1.0, 0, 0], (N, 1)),
                  states=np.zeros((N, 1), np.int64), marks=np.zeros((N, 1), np.int64))
    sim.set_field(0, field_params(field_kind=2, nxyz=(n,) * 3, widths=(width,) * 3, n_binders=1, bead_vol=500.0,
                                  pref=[0.0], intra=[0.0]))
    sim.deposit(-1)
    np.testing.assert_array_equal(sim.density(0)[:, 0], _grid(r, n, width, dtype))
