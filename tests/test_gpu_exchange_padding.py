"""The exchange's row operand is read up to K only.

The rows of the prepared rot_chol pieces are padded to 64 values.  Filling the padding with
NaN changes no bit of the energies, for K tails of 1 to 15 values in a 16-wide step."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

MARK = 0.7109375  # exact in bf16: the low piece is zero


def _poison(prepared, norb, rows):
    """NaN into the padding of both rot_chol pieces; returns how many values."""
    p = prepared.view(torch.bfloat16)
    ld = (norb + 63) // 64 * 64
    head = p[: p.numel() - ld] == MARK
    run = head[:-ld].clone()
    for i in (1, norb - 1, ld):  # a row's first values, its last, the next row's first
        run &= head[i: i + run.numel()]
    for i in (norb, ld - 1):
        run &= p[i: i + run.numel()] == 0.0
    start = int(torch.nonzero(run)[0])
    piece = ((rows * ld + 3) // 4 + 31) // 32 * 32 * 4
    for first in (start, start + piece):
        q = p[first: first + rows * ld].view(rows, ld)
        assert bool((q[:, norb:] == 0.0).all()) and bool((q[:, :norb] == (MARK if first == start else 0.0)).all())
        q[:, norb:] = float("nan")
    return 2 * rows * (ld - norb)


@pytest.mark.parametrize("norb,no", [(17, 5), (20, 5), (31, 12), (40, 34), (200, 40), (203, 36)])
def test_padding_is_not_read(norb, no):
    from ad_afqmc_b200 import propagation, wavefunctions
    from ad_afqmc_b200.walkers import RHFWalkers

    W, G = 5, 7
    trial = wavefunctions.rhf(norb, (no, no))
    wave = {"mo_coeff": np.eye(norb, no)}
    ham = {"h0": 0.0, "chol": np.zeros((G, norb * norb)), "rot_h1": np.zeros((no, norb)),
           "rot_chol": np.full((G, no, norb), MARK), "exp_h1": np.eye(norb), "mf_shifts": np.zeros(G, complex),
           "h0_prop": 0.0}
    prop = propagation.propagator_afqmc(dt=0.005, n_walkers=W, precision="mixed", walker_type="restricted")
    eng = prop.engine(ham, trial, wave)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(2)
    w = torch.eye(norb, no, dtype=torch.complex128, device="cuda") + 0.1 * torch.randn(
        W, norb, no, dtype=torch.complex128, device="cuda", generator=gen)
    e = trial.calc_energy(RHFWalkers(w.clone()), ham, wave, engine=eng)
    assert torch.isfinite(torch.view_as_real(e)).all()
    assert _poison(eng.prepared, norb, G * no) > 0
    assert torch.equal(trial.calc_energy(RHFWalkers(w.clone()), ham, wave, engine=eng), e)
