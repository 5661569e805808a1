"""FP64 contractions at the edges of their tiles.

Sizes just below, at and above the row and column tiles of the force bias, VHS,
propagator and exchange kernels, odd leading dimensions, K tails, one walker.
Reference: the NumPy oracle (1e-10 relative, the FP64 path's parity tolerance).
A pass repeated on the same inputs has to give the same bits: a shared-memory
stage refilled under a warp's reads shows up as a rare difference there."""

import numpy as np
import pytest
import torch

from ad_afqmc_b200.synthetic import make_system
from tests._helpers import device_system, near_trial_walkers, oracle_system, rel_err

pytestmark = pytest.mark.gpu

CASES = [
    # norb, (na, nb), nchol, walkers, trial
    (7, (1, 1), 5, 1, "uhf"),
    (16, (8, 7), 33, 17, "uhf"),
    (33, (9, 8), 65, 40, "uhf"),
    (64, (16, 16), 97, 65, "rhf"),
    (95, (23, 23), 131, 161, "rhf"),
    (97, (25, 24), 129, 33, "uhf"),
    (129, (41, 33), 64, 9, "uhf"),
    (160, (56, 57), 31, 5, "uhf"),
    (225, (64, 48), 17, 3, "uhf"),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: f"n{c[0]}_{c[1][0]}_{c[1][1]}")
def test_f64_step_and_energy_at_tile_edges(case):
    from ad_afqmc_b200.walkers import RHFWalkers, UHFWalkers

    norb, nelec, nchol, W, tr = case
    wt = "restricted" if tr == "rhf" else "unrestricted"
    sys_ = make_system(norb, nelec, nchol, seed=31, trial=tr, chol_scale=0.2)
    rng = np.random.default_rng(5)
    mos = [sys_.mo_coeff] if tr == "rhf" else sys_.mo_coeff
    wk = [near_trial_walkers(rng, m, W, eps=0.5 / np.sqrt(norb)) for m in mos]
    fields = rng.standard_normal((W, nchol))
    o_trial, o_ham, o_wave, o_prop = oracle_system(sys_, wt, 0.005)
    o_prop.n_walkers = W
    init = wk[0] if tr == "rhf" else wk

    def copy():
        return RHFWalkers(wk[0].copy()) if tr == "rhf" else UHFWalkers([w.copy() for w in wk])

    o_pd = o_prop.init_prop_data(o_trial, o_wave, o_ham,
                                 init_walkers=init.copy() if tr == "rhf" else [w.copy() for w in wk])
    o_e = o_trial.calc_energy(init, o_ham, o_wave)
    o_fb = o_trial.calc_force_bias(init, o_ham, o_wave)
    o_pd = o_prop.propagate_constrained(o_trial, o_ham, o_pd, fields, o_wave)
    d_trial, d_ham, d_wave, d_prop, _ = device_system(sys_, wt, 0.005, W)
    assert rel_err(d_trial.calc_energy(copy(), d_ham, d_wave).cpu().numpy(), o_e) < 1e-10
    assert rel_err(d_trial.calc_force_bias(copy(), d_ham, d_wave).cpu().numpy(), o_fb) < 1e-10
    first = None
    for _ in range(20):
        pd = d_prop.init_prop_data(d_trial, d_wave, d_ham, 0, init_walkers=copy())
        pd = d_prop.propagate_constrained(d_trial, d_ham, pd, fields, d_wave)
        got = pd["walkers"].data if isinstance(pd["walkers"].data, list) else [pd["walkers"].data]
        if first is None:
            first = [t.clone() for t in got]
            ref = o_pd["walkers"] if isinstance(o_pd["walkers"], list) else [o_pd["walkers"]]
            for t, r in zip(got, ref):
                assert rel_err(t.cpu().numpy(), r) < 1e-10
            assert rel_err(pd["weights"].cpu().numpy(), o_pd["weights"]) < 1e-9
        for t, f in zip(got, first):
            assert torch.equal(t, f)
