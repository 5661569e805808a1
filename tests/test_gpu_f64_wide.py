"""FP64 VHS and propagator of a basis whose N^2 columns exceed 2^24 (N > 4096).

One Cholesky vector, one walker, so the system fits easily.  Reference: the
Taylor series of VHS = i sqrt(dt) x L on the walker in plain torch (FP64);
tolerance 1e-12 relative, a few hundred eps for sums of 4100 terms."""

import ctypes as C
import math

import pytest
import torch

from ad_afqmc_b200 import _lib

pytestmark = pytest.mark.gpu


def test_trotter_step_beyond_4096_orbitals():
    from ad_afqmc_b200 import wavefunctions
    from ad_afqmc_b200._engine import Engine, dims_for

    norb, dt, terms = 4100, 0.01, 6
    gen = torch.Generator(device="cuda")
    gen.manual_seed(3)
    chol = torch.randn(norb, norb, dtype=torch.float64, device="cuda", generator=gen)
    chol = (chol + chol.T) / math.sqrt(8.0 * norb)
    w = torch.randn(1, norb, 1, dtype=torch.complex128, device="cuda", generator=gen)
    trial = wavefunctions.rhf(norb, (1, 1))
    mo = torch.zeros(norb, 1, dtype=torch.float64, device="cuda")
    mo[0, 0] = 1.0
    ham = {"h0": 0.0, "chol": chol.reshape(1, -1), "rot_h1": torch.zeros(1, norb, dtype=torch.float64),
           "rot_chol": chol[:1].reshape(1, 1, norb).clone(), "exp_h1": torch.eye(norb, dtype=torch.float64),
           "mf_shifts": torch.zeros(1, dtype=torch.complex128), "h0_prop": 0.0}
    d = dims_for(trial, "restricted", 1, 1, "fp64", dt, terms)
    eng = Engine(d, ham, trial, {"mo_coeff": mo})
    x = torch.full((1, 1), 1.7, dtype=torch.float64, device="cuda")
    got = w.clone()
    p, wk, wb = eng.handle
    _lib.check(_lib.lib().afq_apply_trotprop(C.byref(d), p, _lib.pair(got.data_ptr()), x.data_ptr(), wk, wb,
                                             _lib.stream_handle()), "afq_apply_trotprop")
    ref, term = w[0].clone(), w[0].clone()
    vhs = 1j * math.sqrt(dt) * 1.7 * chol
    for n in range(1, terms):
        term = vhs @ term / n
        ref = ref + term
    assert float((got[0] - ref).norm() / ref.norm()) < 1e-12
