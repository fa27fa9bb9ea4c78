"""The chi-free sum S of the exchange (its own kernel) is the energies' S bit for bit,
also where a voxel's bead column fits the integer sums (below 4,096 beads) and a
binder column does not.  S is read from the energy change of an accepted swap of
chi 0 and 1, which the saved state holds."""
import numpy as np
import pytest

from chromo_gb300 import _native as nat
from chromo_gb300.device import binding_params, field_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fp64", [False, True])
@pytest.mark.parametrize("seed", range(4))
def test_exchange_takes_the_energies_sum(seed, fp64):
    rng = np.random.default_rng(seed)
    n, dims, d = 64000, (16, 16, 64), 40.0
    # every bead in one of four cells above each other: ~2,000 beads on each of
    # their voxels, eight layers of which a thread of the sums takes
    cell = np.stack([np.full(n, 4.0), np.full(n, 5.0), 2.0 * (np.arange(n) // 16000)], 1)
    sim = nat.Sim([n, n], [dims, dims], 3, pos_fp64=fp64)
    for rep in range(2):
        r = (cell + 0.5 + rng.uniform(0.05, 0.95, (n, 3)) - 0.5 * np.array(dims)) * d
        sim.set_chain(rep, r=r, t3=np.tile([1.0, 0, 0], (n, 1)), t2=np.tile([0, 1.0, 0], (n, 1)),
                      states=np.full((n, 3), 3), marks=np.zeros((n, 3), np.int64))
        sim.set_field(rep, field_params(field_kind=2, nxyz=dims, widths=tuple(d * k for k in dims), n_binders=3,
                                        chi=0.0, vf_limit=1e9, bead_vol=523.6, pref=[-1.0] * 3, intra=[0.0] * 3))
        sim.set_binding(rep, binding_params(sites=[3] * 3, e_mod=[0.0] * 3, e_nomod=[0.0] * 3, mu=[0.0] * 3))
    sim.deposit(-1)
    S = sim.energies()[:, 4]
    # the smaller S at chi 0: exp((0 - 1) (S_0 - S_1)) >= 1, so the swap is taken
    low = int(S[1] < S[0])
    sim.set_field(1 - low, field_params(field_kind=2, nxyz=dims, widths=tuple(d * k for k in dims), n_binders=3,
                                        chi=1.0, vf_limit=1e9, bead_vol=523.6, pref=[-1.0] * 3, intra=[0.0] * 3))
    sim.deposit(-1)
    sim.exchange(2, 0, 1)
    sim.sync()
    assert sim.chi()[low] == 1.0
    image = sim.save_state().tobytes()
    sim.close()
    assert S[low].tobytes() in image           # (1 - 0) S
    assert (-S[1 - low]).tobytes() in image    # (0 - 1) S
