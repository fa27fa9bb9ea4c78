"""cg_set_chains / cg_get_chains with host arrays that start anywhere within a
128-byte line: the transfer kernels walk the arrays from the line's start, so
the elements before an array, and those after it, must be neither read into the
chain nor written."""
import numpy as np
import pytest

from chromo_gb300 import _native as nat

GUARD = -7


def _placed(shape, dtype, lead, guard=GUARD):
    """An array of ``shape`` that starts ``lead`` elements after a line's start,
    and the guarded buffer that holds it."""
    size = int(np.prod(shape))
    buf = np.full(size + 64, guard, dtype=dtype)
    at = (-(buf.ctypes.data // 8)) % 16 + lead
    part = buf[at:at + size].reshape(shape)
    assert (part.ctypes.data // 8) % 16 == lead
    return part, buf


@pytest.mark.gpu
@pytest.mark.parametrize("fp64", [False, True])
@pytest.mark.parametrize("nb", [1, 3])
def test_any_start_within_a_line(fp64, nb):
    lengths = [4, 5, 6, 11, 16, 43, 86, 5462, 5463]  # 5,462 beads: 64 blocks x 256 threads are 16,384 elements
    rng = np.random.default_rng(11)
    sim = nat.Sim(lengths, [(2, 2, 2)] * len(lengths), nb, pos_fp64=fp64, max_tangent=4)
    cast = np.float64 if fp64 else np.float32
    try:
        for lead in range(16):
            up, out, bufs = [], [], []
            for k, n in enumerate(lengths):
                c = {}
                for j, key in enumerate(("r", "t3", "t2")):
                    # the elements around an upload are not finite: reading them would refuse it
                    c[key], _ = _placed((n, 3), np.float64, (lead + k + j) % 16, guard=np.nan)
                    c[key][:] = rng.normal(size=(n, 3))
                c["states"], _ = _placed((n, nb), np.int64, (lead + 3 * k) % 16, guard=99)
                c["states"][:] = rng.integers(0, 3, size=(n, nb))
                up.append(c)
                parts = [_placed((n, 3), np.float64, (lead + 5 * k + j) % 16) for j in range(3)]
                parts.append(_placed((n, nb), np.int64, (lead + 7 * k) % 16))
                out.append(tuple(p for p, _ in parts))
                bufs.append([b for _, b in parts])
            sim.set_chains(up)
            sim.get_chains(out)
            for c, o, b in zip(up, out, bufs):
                for key, a in zip(("r", "t3", "t2"), o):
                    np.testing.assert_array_equal(a, c[key].astype(cast).astype(np.float64))
                np.testing.assert_array_equal(o[3], c["states"])
                for a, whole in zip(o, b):
                    assert np.count_nonzero(whole == GUARD) >= whole.size - a.size
                    a[...] = GUARD
                    assert np.all(whole == GUARD)
    finally:
        sim.close()
