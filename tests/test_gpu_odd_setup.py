"""Set-up of an unrestricted solve over an odd number of orbitals without given walkers.

The second spin's density matrix then starts 8 bytes off a 16-byte boundary.  The walkers
span the trial's occupied space and their energy is the oracle's (FP64 parity)."""

import numpy as np
import pytest
import torch

from ad_afqmc_b200.synthetic import make_system
from oracle import afqmc_oracle as orc
from tests._helpers import device_system, oracle_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("norb,nelec", [(5, (2, 1)), (37, (9, 8)), (91, (20, 17))])
def test_odd_unrestricted_setup(norb, nelec):
    sys_ = make_system(norb, nelec, 3 * norb, seed=8, trial="uhf", chol_scale=0.3)
    o_trial, o_ham, o_wave, _ = oracle_system(sys_, "unrestricted", 0.005)
    d_trial, d_ham, d_wave, d_prop, _ = device_system(sys_, "unrestricted", 0.005, 3)
    d_wave["rdm1"] = torch.as_tensor(np.asarray(o_trial.rdm1(o_wave)), device="cuda").contiguous()
    pd = d_prop.init_prop_data(d_trial, d_wave, d_ham, 1)
    assert np.allclose(np.abs(pd["overlaps"].cpu().numpy()), 1.0, atol=1e-12)
    e_o = np.real(o_trial.calc_energy(orc.get_init_walkers(o_trial, o_wave, 3, "unrestricted"), o_ham, o_wave))
    assert abs(float(pd["e_estimate"]) - e_o.mean()) < 1e-9 * max(1.0, abs(e_o.mean()))
