"""The one-kernel FP64 step of small systems against the NumPy oracle.

One orbital up to the kernel's limit and just beyond it, every trial and walker
type, one to six Taylor terms, one walker to more than a wave; three steps in a
row, so that the second and third start from the Green's function the first left.
Tolerance: the FP64 path's 1e-10 relative (weights 1e-9: three steps of the
logarithm of the total weight over dt)."""

import numpy as np
import pytest

from ad_afqmc_b200.synthetic import make_system
from oracle import afqmc_oracle as orc
from tests._helpers import device_system, near_trial_walkers, rel_err

pytestmark = pytest.mark.gpu

CASES = [
    # norb, (na, nb), nchol, walkers, trial, walker type, Taylor terms
    (1, (1, 1), 1, 1, "rhf", "restricted", 6),
    (2, (1, 2), 3, 5, "uhf", "unrestricted", 2),
    (6, (3, 3), 15, 50, "uhf", "unrestricted", 6),
    (10, (5, 5), 50, 100, "rhf", "restricted", 6),
    (11, (4, 4), 33, 7, "rhf", "unrestricted", 1),
    (16, (8, 7), 97, 3, "uhf", "unrestricted", 4),
    (17, (17, 17), 20, 9, "rhf", "restricted", 6),
    (20, (9, 8), 130, 301, "uhf", "unrestricted", 6),
    (24, (12, 12), 61, 148, "rhf", "restricted", 6),
    (24, (12, 12), 61, 149, "rhf", "restricted", 6),   # beyond the rule: the tensor-core launches
    (25, (6, 5), 31, 12, "uhf", "unrestricted", 6),    # likewise
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: f"n{c[0]}_w{c[3]}_{c[4]}_{c[5]}_t{c[6]}")
def test_three_steps(case):
    from ad_afqmc_b200.walkers import RHFWalkers, UHFWalkers

    norb, nelec, nchol, W, tr, wt, terms = case
    sys_ = make_system(norb, nelec, nchol, seed=41, trial=tr, chol_scale=0.2)
    rng = np.random.default_rng(6)
    mos = sys_.mo_coeff if tr == "uhf" else [sys_.mo_coeff] * (1 if wt == "restricted" else 2)
    wk = [near_trial_walkers(rng, m, W, eps=0.3 / np.sqrt(norb)) for m in mos]
    fields = rng.standard_normal((3, W, nchol))
    o_trial = orc.RHFTrial(norb, nelec) if tr == "rhf" else orc.UHFTrial(norb, nelec)
    o_wave = sys_.wave_data()
    o_prop = orc.Propagator(dt=0.005, n_walkers=W, n_exp_terms=terms, walker_type=wt)
    o_ham = o_trial.build_measurement_intermediates(sys_.ham_data(), o_wave)
    o_ham = o_prop.build_propagation_intermediates(o_ham, o_trial, o_wave)
    init = [w.copy() for w in wk]
    o_pd = o_prop.init_prop_data(o_trial, o_wave, o_ham, init_walkers=init[0] if len(init) == 1 else init)
    d_trial, d_ham, d_wave, d_prop, _ = device_system(sys_, wt, 0.005, W, n_exp_terms=terms)
    own = [w.copy() for w in wk]
    pd = d_prop.init_prop_data(d_trial, d_wave, d_ham, 0,
                               init_walkers=RHFWalkers(own[0]) if len(own) == 1 else UHFWalkers(own))
    for f in fields:
        if terms == 1:  # the oracle's empty Taylor sum: the two half-steps alone
            o_prop.apply_trotprop_single_det_vhs = lambda w, v, e: e @ (e @ w)
        o_pd = o_prop.propagate_constrained(o_trial, o_ham, o_pd, f, o_wave)
        pd = d_prop.propagate_constrained(d_trial, d_ham, pd, f, d_wave)
        ref = o_pd["walkers"] if isinstance(o_pd["walkers"], list) else [o_pd["walkers"]]
        got = pd["walkers"].data if isinstance(pd["walkers"].data, list) else [pd["walkers"].data]
        for g, r in zip(got, ref):
            assert rel_err(g.cpu().numpy(), r) < 1e-10
        assert rel_err(pd["overlaps"].cpu().numpy(), o_pd["overlaps"]) < 1e-10
        assert rel_err(pd["weights"].cpu().numpy(), o_pd["weights"]) < 1e-9
