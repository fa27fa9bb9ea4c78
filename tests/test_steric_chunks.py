"""The split of a chain into the steric kernels' tiles and chunks, for chains of two
beads to the longest accepted (2e9): the chunks cover the chain, fit the grid's y
axis (65,535) and the buffer of the tiles' sums (n_beads + 32); and on the GPU one
moved bead of a chain beyond 65,535 chunks of 256 columns."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

HDR = Path(__file__).resolve().parents[1] / "chromo_gb300" / "csrc" / "cg_steric_tiles.h"


@pytest.fixture(scope="module")
def chunk(tmp_path_factory):
    d = tmp_path_factory.mktemp("steric")
    (d / "t.c").write_text(f'#include "{HDR}"\nlong long chunk(long long n, long long m, int sm, int* rows)'
                           "{ return cg_steric_split(n, m, sm, rows); }\n")
    subprocess.check_call(["gcc", "-O1", "-shared", "-fPIC", "-o", str(d / "t.so"), str(d / "t.c")])
    f = ctypes.CDLL(str(d / "t.so")).chunk
    f.argtypes = [ctypes.c_longlong, ctypes.c_longlong, ctypes.c_int, ctypes.c_void_p]
    f.restype = ctypes.c_longlong
    return f


@pytest.mark.parametrize("n", [2, 255, 256, 257, 1025, 10000, 32769, 1000000, 16776960, 16776961, 2000000000])
def test_chunks_fit_the_grid_and_the_sums(chunk, n):
    for m in sorted({1, 32, 33, 288, 289, 320, n}):
        if m > n:
            continue
        rows = ctypes.c_int()
        c = chunk(n, m, 152, ctypes.byref(rows))
        tiles, chunks = (m + rows.value - 1) // rows.value, (n + c - 1) // c
        assert rows.value in (1, 2, 4, 8, 16, 32)
        assert c % 256 == 0 and (c == 256 or c >= 1024)
        assert chunks <= 65535 and tiles <= 2 ** 31 - 1
        assert tiles * chunks <= n + 32


@pytest.mark.gpu
def test_one_moved_bead_of_a_very_long_chain():
    from chromo_gb300 import _native as nat
    from oracle import oracle as orc
    n = 16777300  # 65,537 chunks of 256 columns
    r = np.zeros((n, 3))  # every coordinate exact in FP32, beads at least 1 apart
    k = np.arange(n)
    far = k >= 2 ** 24
    r[:, 0] = np.where(far, k // 2 * 2, k)
    r[:, 1] = np.where(far, k % 2, 0)
    sim = nat.Sim([n], [[1, 1, 1]], 1)
    sim.set_chain(0, r=r)
    for i in (0, n // 2, n - 1):
        trial = r[i:i + 1] + [[0.0, 0.0, 0.5]]
        got, want = sim.steric_delta(0, i, i + 1, trial, 2.5), orc.steric_delta(r, trial, i, i + 1, 2.5)
        assert want != 0.0
        # at most 16 terms of at most 2.5^12 + 2 2.5^6 + 1 each, in another order
        assert abs(got - want) <= 1e-12 * 16 * (2.5 ** 6 + 1) ** 2, (i, got, want)
    sim.close()
