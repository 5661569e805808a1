"""The mixed exchange's sums over rows and Cholesky vectors are FP64 sums.

Row products whose sum cancels to 1 across 52 bits: exact in FP64 in any order, not
in fewer bits.  A walker whose rows overflow FP32 has an infinite energy (not
NaN), which the block average clamps to its estimate."""

import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

DT = 0.005


def _system(mo, W, rot_chol, precision):
    from ad_afqmc_b200 import propagation, wavefunctions

    (norb, no), G = mo.shape, rot_chol.shape[0]
    trial = wavefunctions.rhf(norb, (no, no))
    wave = {"mo_coeff": mo}
    ham = {"h0": 0.0, "chol": np.zeros((G, norb * norb)), "rot_h1": np.zeros((no, norb)), "rot_chol": rot_chol,
           "exp_h1": np.eye(norb), "mf_shifts": np.zeros(G, complex), "h0_prop": 0.0}
    prop = propagation.propagator_afqmc(dt=DT, n_walkers=W, precision=precision, walker_type="restricted")
    return trial, wave, ham, prop, prop.engine(ham, trial, wave)


@pytest.mark.parametrize("precision", ["mixed", "mixed_hi"])
@pytest.mark.parametrize("no", [10, 17, 28, 40, 48], ids=lambda n: f"no{n}")
def test_row_sums_keep_fp64(no, precision):
    """f = rot_chol's occupied block (Theta = [1; 0]): pairs f_ij f_ji of +2^51, +2^26, +1,
    -2^51 and -2^26, each in two rows."""
    from ad_afqmc_b200.walkers import RHFWalkers

    norb, W, G = no + 9, 3, 130
    rc = np.zeros((G, no, norb))
    for g in (0, 64, G - 1):
        for p, (a, b) in enumerate([(26, 25), (13, 13), (0, 0), (26, 25), (13, 13)]):
            sign = 1.0 if p < 3 else -1.0
            rc[g, 2 * p, 2 * p + 1], rc[g, 2 * p + 1, 2 * p] = 2.0**a, sign * 2.0**b
    trial, wave, ham, _, eng = _system(np.eye(norb, no), W, rc, precision)
    w = torch.eye(norb, no, dtype=torch.complex128, device="cuda").repeat(W, 1, 1)
    e = trial.calc_energy(RHFWalkers(w), ham, wave, engine=eng)
    assert torch.equal(e.cpu(), torch.full((W,), -3 * 2.0, dtype=torch.complex128))


@pytest.mark.parametrize("precision", ["mixed", "mixed_hi"])
@pytest.mark.parametrize("no", [3, 10, 40], ids=lambda n: f"no{n}")
def test_overflowed_rows_stay_infinite(no, precision):
    """The second walker is all but orthogonal to the trial: its Theta has one entry of
    1e20, so f_00^2 leaves FP32's range in every row tile.  (The trial occupies rows
    1 .. no: the QR keeps the entry of 1e-20 below the pivot.)"""
    from ad_afqmc_b200 import _lib
    from ad_afqmc_b200.propagation import make_state
    from ad_afqmc_b200.walkers import RHFWalkers

    norb, W, G = no + 5, 3, 140
    rc = 1e-3 * np.random.default_rng(4).standard_normal((G, no, norb))
    rc[:, :, 0] = 0.0
    rc[:, 0, 0] = 1.0
    mo = np.eye(norb, no, -1)
    trial, wave, ham, prop, eng = _system(mo, W, rc, precision)
    w = torch.from_numpy(mo + 0j).cuda().repeat(W, 1, 1)
    w[1, 1, 0] = 1e-20
    w[1, 0, 0] = 1.0
    e = trial.calc_energy(RHFWalkers(w.clone()), ham, wave, engine=eng).cpu().numpy()
    f = rc @ mo
    ref = 2 * (np.einsum("gii->g", f) ** 2).sum() - np.einsum("gij,gji->", f, f)
    assert np.isinf(e[1].real) and not np.isnan(e[1].imag)
    assert np.allclose(e[[0, 2]], ref, rtol=1e-4, atol=1e-9)
    # the block's energy: the infinite one is clamped to the estimate
    pd = prop.init_prop_data(trial, wave, dict(ham, e_estimate=0.0), 0, init_walkers=RHFWalkers(w))
    out = torch.zeros(2, dtype=torch.float64, device="cuda")
    st = make_state(pd)
    p, wk, wb = eng.handle
    _lib.check(_lib.lib().afq_block_end(C.byref(eng.dims), p, C.byref(st), out.data_ptr(), wk, wb,
                                        _lib.stream_handle()), "afq_block_end")
    assert torch.isfinite(out).all()
