"""FP64 exchange and orbital energy over every tile width and walkers per tile.

One to 64 electrons per spin, tiles of several walkers whose columns end inside and
at the end of an MMA tile, ragged last tiles of walkers and of Cholesky vectors, odd
basis sizes, few walkers (one per tile) and many.  Reference: the NumPy oracle (1e-10
relative, the FP64 path's parity tolerance); repeated passes give the same bits."""

import numpy as np
import pytest
import torch

from ad_afqmc_b200.synthetic import make_system
from tests._helpers import device_system, near_trial_walkers, oracle_system, rel_err

pytestmark = pytest.mark.gpu

CASES = [
    # norb, (na, nb), nchol, walkers
    (9, (1, 2), 700, 150),
    (12, (3, 4), 300, 333),
    (15, (5, 6), 131, 200),
    (17, (7, 8), 257, 3),
    (24, (9, 10), 90, 161),
    (30, (11, 12), 61, 130),
    (33, (14, 13), 40, 150),
    (31, (15, 16), 77, 100),
    (40, (17, 21), 23, 160),
    (29, (26, 27), 45, 90),
    (41, (25, 28), 17, 31),
    (66, (41, 49), 9, 5),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: f"n{c[0]}_{c[1][0]}_{c[1][1]}_w{c[3]}")
def test_energy(case):
    from ad_afqmc_b200.walkers import UHFWalkers

    norb, nelec, nchol, W = case
    sys_ = make_system(norb, nelec, nchol, seed=29, trial="uhf", chol_scale=0.3)
    rng = np.random.default_rng(11)
    wk = [near_trial_walkers(rng, m, W, eps=0.5 / np.sqrt(norb)) for m in sys_.mo_coeff]
    o_trial, o_ham, o_wave, _ = oracle_system(sys_, "unrestricted", 0.005)
    d_trial, d_ham, d_wave, _, _ = device_system(sys_, "unrestricted", 0.005, W)
    ref = o_trial.calc_energy(wk, o_ham, o_wave)
    e = [d_trial.calc_energy(UHFWalkers([w.copy() for w in wk]), d_ham, d_wave) for _ in range(5)]
    assert rel_err(e[0].cpu().numpy(), ref) < 1e-10
    assert all(torch.equal(e[0], x) for x in e[1:])


@pytest.mark.parametrize("norb,no,nchol,W", [(9, 1, 300, 70), (20, 5, 50, 40), (27, 10, 33, 9), (30, 26, 20, 12)])
def test_orbital_energy(norb, no, nchol, W):
    """f = rot_chol's virtual columns times Theta's virtual rows; 2 c s1 - s2 summed."""
    from ad_afqmc_b200 import hamiltonian, wavefunctions
    from ad_afqmc_b200.walkers import RHFWalkers

    sys_ = make_system(norb, (no, no), nchol, seed=3, trial="rhf", chol_scale=0.3)
    rng = np.random.default_rng(8)
    w = near_trial_walkers(rng, sys_.mo_coeff, W, eps=0.3 / np.sqrt(norb))
    prj = rng.standard_normal((2, no))
    trial = wavefunctions.rhf_lno(norb, (no, no))
    wave = dict(sys_.wave_data(), prjlo=prj)
    ham = hamiltonian.hamiltonian(norb).build_measurement_intermediates(sys_.ham_data(), trial, wave)
    got = trial.calc_orbenergy(RHFWalkers(w.copy()), ham, wave).cpu().numpy()
    mo, L = sys_.mo_coeff, np.asarray(sys_.ham_data()["chol"]).reshape(nchol, norb, norb)
    theta = w @ np.linalg.inv(mo.T @ w)
    f = np.einsum("gip,wpj->wgij", np.einsum("pi,gpq->giq", mo, L)[:, :, no:], theta[:, no:], optimize=True)
    m = prj.T @ prj
    c, s1 = np.einsum("wgii->wg", f), np.einsum("wgij,ij->wg", f, m)
    s2 = np.einsum("wgij,wgjk,ik->wg", f, f, m, optimize=True)
    assert rel_err(got, (2 * c * s1 - s2).sum(1)) < 1e-10
