"""S = C^T W, its inverse and Theta at the edges of the kernels' tiles.

Occupations around every change of the launch (32, 40, 48, 64), of the row tiles that a
smaller sector works on (16, 32) and of the k-steps, orbitals around the chunks of 32 rows
with each remainder of four.  calc_green runs the one-kernel form; the FP64 force
bias of more than 24 orbitals the three-kernel form.  Tolerance: 200 eps times the largest
condition number of the overlap matrices."""

import numpy as np
import pytest

from ad_afqmc_b200.synthetic import make_system
from tests._helpers import device_system, near_trial_walkers, rel_err

pytestmark = pytest.mark.gpu

CASES = [
    (25, (1, 1)), (27, (3, 2)), (31, (16, 17)), (32, (32, 9)), (33, (8, 33)), (41, (40, 15)),
    (64, (41, 16)), (65, (47, 48)), (66, (49, 5)), (97, (64, 63)), (130, (24, 40)), (159, (39, 2)),
]


@pytest.mark.parametrize("norb,nelec", CASES, ids=lambda v: str(v).replace(" ", ""))
def test_green_and_force_bias(norb, nelec):
    from ad_afqmc_b200.walkers import UHFWalkers

    W, nchol = 6, 3
    sys_ = make_system(norb, nelec, nchol, seed=9, trial="uhf", chol_scale=0.2)
    rng = np.random.default_rng(norb)
    wk = [near_trial_walkers(rng, m, W, eps=0.3 / np.sqrt(norb)) for m in sys_.mo_coeff]
    trial, ham, wave, _, _ = device_system(sys_, "unrestricted", 0.005, W)
    walkers = UHFWalkers([w.copy() for w in wk])
    greens, fb, ov, cond = [], 0.0, 1.0, 1.0
    for c, w in zip(sys_.mo_coeff, wk):
        c = np.asarray(c)[:, : w.shape[2]]
        s = np.einsum("pi,wpj->wij", c, w)
        theta = np.einsum("wpj,wji->wpi", w, np.linalg.inv(s))
        cond = max(cond, np.linalg.cond(s).max())
        ov = ov * np.linalg.det(s)
        greens.append(theta.transpose(0, 2, 1))
        rot = np.einsum("pi,gpq->giq", c, np.asarray(sys_.ham_data()["chol"]).reshape(nchol, norb, norb))
        fb = fb + np.einsum("giq,wqi->wg", rot, theta)
    tol = 200 * np.finfo(float).eps * cond
    got = trial.calc_green(walkers, wave)
    for g, ref in zip(got, greens):
        assert rel_err(g.cpu().numpy(), ref) < tol
    assert rel_err(trial.calc_overlap(walkers, wave).cpu().numpy(), ov) < max(nelec) * tol
    assert rel_err(trial.calc_force_bias(walkers, ham, wave).cpu().numpy(), fb) < 10 * tol
