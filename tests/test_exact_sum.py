"""The fixed-point sum of FP64 terms (cg_exact.h, compiled here) against math.fsum,
which rounds the exact sum once: terms over the whole range, of both signs, cancelling
to the last bit, single ones, and as many as the limbs hold between two carries, in any
order; and the terms that are left to the caller.  On the GPU: the field dE of FP64
moves, in the CTA's pooled table, in their own and overflowing from one to the other,
is the same for any number of warps."""
import ctypes
import math
import subprocess
from pathlib import Path

import numpy as np
import pytest

HDR = Path(__file__).resolve().parents[1] / "chromo_gb300" / "csrc" / "cg_exact.h"


@pytest.fixture(scope="module")
def exact(tmp_path_factory):
    d = tmp_path_factory.mktemp("exact")
    (d / "x.c").write_text(
        f'#include "{HDR}"\n'
        "double total(const double* x, long n, long* left) { int L[CGX_LIMBS] = {0}, v[4]; long room = CGX_TERMS;\n"
        "  *left = 0;\n"
        "  for (long j = 0; j < n; j++) { unsigned long long b; memcpy(&b, x + j, 8);\n"
        "    const int i = cgx_split(b, v);\n"
        "    if (i < 0) { ++*left; continue; }\n"
        "    for (int k = 0; k < 4; k++) L[i + k] += v[k];\n"
        "    if (--room == 0) { cgx_carry(L); room = CGX_TERMS; } }\n"
        "  return cgx_value(L); }\n")
    subprocess.check_call(["gcc", "-O2", "-ftrapv", "-shared", "-fPIC", "-o", str(d / "x.so"), str(d / "x.c")])
    f = ctypes.CDLL(str(d / "x.so")).total
    f.argtypes = [ctypes.c_void_p, ctypes.c_long, ctypes.c_void_p]
    f.restype = ctypes.c_double

    def total(x):
        x = np.ascontiguousarray(x, dtype=np.float64)
        left = ctypes.c_long()
        return f(x.ctypes.data, len(x), ctypes.byref(left)), left.value
    return total


def test_sum_is_the_exact_sum_rounded_once(exact):
    rng = np.random.default_rng(5)
    sets = [rng.normal(size=n) for n in (1, 2, 33, 2047, 2048, 50000)]
    sets += [rng.normal(size=300) * 2.0 ** rng.integers(-100, 28, 300) for _ in range(300)]
    sets += [s * 2.0 ** float(rng.integers(-90, 20)) for s in rng.normal(size=(300, 40))]
    big = np.full(2047, np.nextafter(2.0 ** 32, 0.0))
    sets += [big, -big, np.full(4094, -(2.0 ** -108)), np.array([2.0 ** 31, -(2.0 ** 31), 2.0 ** -108]),
             np.array([1.0, 2.0 ** -53, 2.0 ** -105]), np.array([1.0, 2.0 ** -53]), np.array([1.0, -(2.0 ** -54)])]
    for x in list(sets):
        y = np.concatenate([x, -x[: len(x) // 2]])
        sets += [rng.permutation(y), np.concatenate([y, -y])]
    for x in sets:
        x = x[(np.abs(x) >= 2.0 ** -108) & (np.abs(x) < 2.0 ** 32)]
        got, left = exact(x)
        assert left == 0 and got == math.fsum(x), (len(x), got, math.fsum(x))


def test_terms_outside_the_range_are_left(exact):
    x = [0.0, -0.0, 2.0 ** 32, -(2.0 ** 32), np.nextafter(2.0 ** -108, 0.0), 5e-324, np.inf, -np.inf, np.nan, 1e300]
    assert exact(x) == (0.0, len(x))
    assert exact(x + [3.5]) == (3.5, len(x))


@pytest.mark.gpu
@pytest.mark.parametrize("n,dims,amp", [(400, (30, 30, 30), 60), (400, (30, 30, 30), 255), (3000, (20, 21, 22), 600),
                                        (500, (8192, 8192, 1), 120), (400, (1, 40, 1), 200), (1200, (40, 40, 40), 1200)])
def test_fp64_energies_do_not_depend_on_warps(n, dims, amp):
    from test_own_table import _sim
    from chromo_gb300.device import move_ctl
    got = []
    for W in (1, 2, 5, 12, 12):
        sim = _sim(n, dims, amp, True, W)
        sim.set_controllers(0, [move_ctl(m, amp_move=0.2 if m != "slide" else 2.0, amp_bead=amp, num_per_cycle=24,
                                         simple=False) for m in ("crank_shaft", "end_pivot", "slide", "change_binding_state")])
        log = sim.run_logged(2, 99, 1000)[0]
        got.append((log["dE_field"].copy(), log["dE_poly"].copy(), sim.energies()[0, 3:4]) + sim.get_chain(0))
        sim.close()
    assert np.count_nonzero(got[0][0]) > 20
    for other in got[1:]:
        for a, b in zip(got[0], other):
            np.testing.assert_array_equal(a, b)
