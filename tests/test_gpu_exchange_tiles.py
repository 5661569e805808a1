"""Exchange on the tensor cores at the edges of its tiles and plans.

Every column width (BN 32 ... 128), one and several walkers per tile, one and
two accumulator buffers, the row operand wholly or partly in TMEM or streamed,
K tails of one to four 16-wide steps, ragged last tiles.  Reference: the NumPy
oracle's local energies; tolerance: the split products' relative accuracy as
in the other mixed-precision tests (BF16x3 1e-4, BF16x6 2e-5)."""

import numpy as np
import pytest
import torch

from ad_afqmc_b200.synthetic import make_system
from tests._helpers import device_system, near_trial_walkers, oracle_system, rel_err

pytestmark = pytest.mark.gpu

TOL = {"mixed": 1e-4, "mixed_hi": 2e-5}

CASES = [
    # norb, (na, nb), nchol, walkers
    (17, (1, 1), 131, 70),     # No = 1: 64 walkers and 128 Cholesky vectors per tile
    (33, (5, 3), 53, 19),      # several walkers per tile, both spins ragged
    (48, (13, 16), 20, 9),     # BN = 80 / 96, K without a tail
    (65, (25, 21), 12, 7),     # BN = 128 with two walkers per tile, a one-step tail
    (97, (33, 40), 11, 5),     # one walker per tile, BN = 80, a partly filled last row tile
    (200, (40, 31), 7, 9),     # low piece partly in TMEM, partly in shared memory
    (120, (48, 64), 5, 3),     # BN = 96 and 128
    (300, (60, 57), 5, 4),     # one accumulator buffer, part of the low piece in shared memory
    (530, (50, 2), 4, 2),      # K too long for TMEM beside BN = 128: both operands stream
]


@pytest.mark.parametrize("precision", ["mixed", "mixed_hi"])
@pytest.mark.parametrize("case", CASES, ids=lambda c: f"n{c[0]}_{c[1][0]}_{c[1][1]}")
def test_energy_at_tile_edges(case, precision):
    from ad_afqmc_b200.walkers import UHFWalkers

    norb, nelec, nchol, W = case
    sys_ = make_system(norb, nelec, nchol, seed=23, trial="uhf", chol_scale=0.25)
    rng = np.random.default_rng(7)
    wk = [near_trial_walkers(rng, m, W, eps=0.5 / np.sqrt(norb)) for m in sys_.mo_coeff]
    o_trial, o_ham, o_wave, _ = oracle_system(sys_, "unrestricted", 0.005)
    d_trial, d_ham, d_wave, d_prop, _ = device_system(sys_, "unrestricted", 0.005, W, precision=precision)
    ref = o_trial.calc_energy(wk, o_ham, o_wave)
    eng = d_prop.engine(d_ham, d_trial, d_wave)
    e = d_trial.calc_energy(UHFWalkers([w.copy() for w in wk]), d_ham, d_wave, engine=eng)
    assert rel_err(e.cpu().numpy(), ref) < TOL[precision]
    again = d_trial.calc_energy(UHFWalkers([w.copy() for w in wk]), d_ham, d_wave, engine=eng)
    assert torch.equal(e, again)
    eng.check_status()
