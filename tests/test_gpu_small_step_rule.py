"""Both FP64 step paths around the line between them, against the oracle.

The one-kernel step with thousands of walkers and with one, the tensor-core launches at the
same basis sizes (many walkers, or too much work per walker for one SM), one walker and
ragged tiles included.  Which path ran is read off the VHS launches.  Tolerance: 1e-10
relative, the FP64 path's parity tolerance; repeated steps give the same bits."""

import numpy as np
import pytest
import torch

from ad_afqmc_b200 import _lib
from ad_afqmc_b200.synthetic import make_system
from tests._helpers import device_system, near_trial_walkers, oracle_system, rel_err

pytestmark = pytest.mark.gpu

CASES = [
    # norb, (na, nb), nchol, walkers, trial, one kernel
    (6, (3, 3), 15, 3000, "uhf", True),
    (10, (5, 5), 40, 2500, "rhf", True),
    (20, (10, 9), 40, 1, "uhf", True),
    (24, (6, 6), 48, 149, "rhf", True),
    (16, (8, 8), 64, 1200, "rhf", False),
    (20, (10, 10), 120, 700, "rhf", False),
    (23, (12, 11), 61, 301, "uhf", False),
    (24, (24, 23), 380, 1, "uhf", False),
    (24, (17, 17), 301, 2, "rhf", False),
    (27, (1, 2), 5, 1, "uhf", False),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: f"n{c[0]}_{c[1][0]}_{c[1][1]}_w{c[3]}")
def test_step(case):
    from ad_afqmc_b200.walkers import RHFWalkers, UHFWalkers

    norb, nelec, nchol, W, tr, one = case
    wt = "restricted" if tr == "rhf" else "unrestricted"
    sys_ = make_system(norb, nelec, nchol, seed=37, trial=tr, chol_scale=0.2)
    rng = np.random.default_rng(6)
    mos = [sys_.mo_coeff] if tr == "rhf" else sys_.mo_coeff
    wk = [near_trial_walkers(rng, m, W, eps=0.5 / np.sqrt(norb)) for m in mos]
    fields = rng.standard_normal((W, nchol))
    o_trial, o_ham, o_wave, o_prop = oracle_system(sys_, wt, 0.005)
    o_prop.n_walkers = W
    o_pd = o_prop.init_prop_data(o_trial, o_wave, o_ham,
                                 init_walkers=wk[0].copy() if tr == "rhf" else [w.copy() for w in wk])
    o_pd = o_prop.propagate_constrained(o_trial, o_ham, o_pd, fields, o_wave)
    ref = o_pd["walkers"] if isinstance(o_pd["walkers"], list) else [o_pd["walkers"]]
    d_trial, d_ham, d_wave, d_prop, _ = device_system(sys_, wt, 0.005, W)
    first = None
    for _ in range(5):
        init = RHFWalkers(wk[0].copy()) if tr == "rhf" else UHFWalkers([w.copy() for w in wk])
        pd = d_prop.init_prop_data(d_trial, d_wave, d_ham, 0, init_walkers=init)
        before = _lib.launch_count("vhs")
        pd = d_prop.propagate_constrained(d_trial, d_ham, pd, fields, d_wave)
        assert (_lib.launch_count("vhs") == before) == one
        got = pd["walkers"].data if isinstance(pd["walkers"].data, list) else [pd["walkers"].data]
        if first is None:
            first = [t.clone() for t in got]
            for t, r in zip(got, ref):
                assert rel_err(t.cpu().numpy(), r) < 1e-10
            assert rel_err(pd["weights"].cpu().numpy(), o_pd["weights"]) < 1e-9
            assert rel_err(pd["overlaps"].cpu().numpy(), o_pd["overlaps"]) < 1e-9
        assert all(torch.equal(t, f) for t, f in zip(got, first))
