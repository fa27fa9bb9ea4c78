"""The sums over a replica's beads and voxels with one to eight CTAs per replica (few
large replicas to many small ones, equal and of very different lengths): the energies
and derivative terms are those of the same chain alone, to rounding (voxel products are
summed exactly, ~100 FP64 additions of the bonds' positive terms); the exchange's S is
the energies' S bit for bit, from its own launch and from the captured rounds, and the
bound sites of a mu ladder's binder are exact."""
import numpy as np
import pytest

from chromo_gb300 import _native as nat
from chromo_gb300 import synthetic as syn
from chromo_gb300.device import binding_params, bonds_array, field_params, move_ctl
from chromo_gb300.energetics import dss_parameters

pytestmark = pytest.mark.gpu


def _states(n, nb=2):
    return np.random.default_rng([n, 1]).integers(0, 3, size=(n, nb))


def _sim(lengths, dims, chi, mu=None, nb=2):
    sim = nat.Sim(lengths, [dims] * len(lengths), nb, max_tangent=8, max_segment=10)
    for rep, n in enumerate(lengths):
        rng = np.random.default_rng(n)  # the same chain for the same length
        r = syn.gaussian_walk(rng, n, 16.5)
        t3, t2 = syn.tangents_from_coordinates(r)
        _, eb, g, ep, epp, eta = dss_parameters(np.full(n - 1, 16.5), 53.0)
        sim.set_chain(rep, r=r, t3=t3, t2=t2, states=_states(n, nb),
                      marks=rng.integers(0, 3, size=(n, nb)), bonds=bonds_array(eb, g, ep, epp, eta))
        sim.set_field(rep, field_params(field_kind=2, nxyz=dims, widths=tuple(40.0 * d for d in dims), n_binders=nb,
                                        chi=float(chi[rep]), vf_limit=0.02, bead_vol=523.6, pref=[-900.0] * nb,
                                        intra=[-3.0] * nb))
        sim.set_binding(rep, binding_params(sites=[2] * nb, e_mod=[-0.01] * nb, e_nomod=[1.52] * nb, 
                                          mu=[-0.4, -0.4 if mu is None else float(mu[rep])]))
        sim.set_controllers(rep, [move_ctl("slide", amp_move=1.0, amp_bead=2, num_per_cycle=1, simple=False, move_on=0)])
    sim.deposit(-1)
    return sim


CASES = [([1500, 1500], (30, 30, 30)), ([900] * 40, (20, 20, 20)), ([600] * 160, (24, 24, 24)),
         ([40] * 400, (5, 6, 7)), ([3000] + [30] * 199, (6, 6, 6))]


@pytest.mark.parametrize("lengths,dims", CASES)
def test_sums_of_a_replica_do_not_depend_on_the_batch(lengths, dims):
    chi = np.where(np.arange(len(lengths)) % 2, 1.0, 0.0)
    sim = _sim(lengths, dims, chi)
    e = sim.energies()
    _, T = sim.gradient(positions=False)
    for rep in (0, 1, len(lengths) - 1):
        alone = _sim([lengths[rep]], dims, [chi[rep]])
        np.testing.assert_allclose(e[rep], alone.energies()[0], rtol=1e-13, atol=1e-10)
        np.testing.assert_allclose(T[rep], alone.gradient(positions=False)[1][0], rtol=1e-13)
        alone.close()
    sim.close()


def _exchange(lengths, dims, chi, mu, captured):
    """S before one exchange round (two rungs; mu rungs where there are grids of
    them), chi and mu after it and the saved state."""
    sim = _sim(lengths, dims, chi, mu)
    sim.set_mu_ladder(2 if len(lengths) % 4 == 0 else 0, 1)
    S = sim.energies()[:, 4]
    if captured:
        sim.run_batched(1, 1, 2, 5)  # its moves are off
    else:
        sim.exchange(2, 0, 5)
    sim.sync()
    out = S, sim.chi(), sim.mu(1), sim.save_state().tobytes()
    sim.close()
    return out


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("lengths,dims", CASES)
def test_exchange_takes_the_energies_sum(lengths, dims, captured):
    chi = np.where(np.arange(len(lengths)) % 2, 1.0, 0.0)
    S, got, _, image = _exchange(lengths, dims, chi, None, captured)
    swapped = np.nonzero(got != chi)[0]
    assert len(swapped)
    for rep in swapped[:8]:
        assert ((got[rep] - chi[rep]) * S[rep]).tobytes() in image


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("lengths,dims", [c for c in CASES if len(c[0]) % 4 == 0])
def test_bound_sites_are_exact(lengths, dims, captured):
    mu = np.where(np.arange(len(lengths)) // 2 % 2, -0.5, -1.0)
    _, _, got, image = _exchange(lengths, dims, np.ones(len(lengths)), mu, captured)
    swapped = np.nonzero(got != mu)[0]
    assert len(swapped)
    for rep in swapped[:8]:
        sites = float(_states(lengths[rep])[:, 1].sum())
        assert np.float64((mu[rep] - got[rep]) * sites).tobytes() in image
