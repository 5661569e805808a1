"""The QR in panels of four reflectors against LAPACK.

Orbitals at and around every change of the rows a lane holds (32, 64, 128, 224,
320) and beyond the last, one column to 64 with each remainder of four, square
walkers, both placements of the walker, a matrix that is triangular already (zero
reflectors).  Tolerance: 50 eps times the batch's largest condition number, the
backward error of Householder QR carried into Q."""

import numpy as np
import pytest

from oracle import afqmc_oracle as orc
from tests._helpers import rel_err

pytestmark = pytest.mark.gpu

CASES = [
    # norb, (na, nb)
    (1, (1, 1)), (3, (2, 1)), (5, (5, 4)), (31, (6, 3)), (32, (32, 7)), (33, (9, 8)),
    (64, (13, 64)), (65, (5, 30)), (128, (17, 2)), (129, (11, 40)), (224, (64, 63)),
    (225, (21, 4)), (300, (1, 47)), (320, (64, 33)), (321, (10, 3)),
]


def _tol(a):
    return 50 * np.finfo(float).eps * np.linalg.cond(a).max()


@pytest.mark.parametrize("qr_mode", [1, 2])
@pytest.mark.parametrize("norb,nelec", CASES, ids=lambda v: str(v).replace(" ", ""))
def test_qr(norb, nelec, qr_mode):
    from ad_afqmc_b200 import _lib
    from ad_afqmc_b200.walkers import RHFWalkers, UHFWalkers, _dims

    rng = np.random.default_rng(norb)
    W = 5
    a, b = (rng.standard_normal((W, norb, k)) + 1j * rng.standard_normal((W, norb, k)) for k in nelec)
    qs, _ = orc.qr_unrestricted([a, b])
    qa, na = orc.qr_restricted(a)
    t = _lib.afq_tuning()
    t.qr_mode = qr_mode
    keys = [_dims(norb, nelec, W, "unrestricted"), _dims(norb, (nelec[0],) * 2, W, "restricted")]
    for d in keys:
        _lib.set_tuning(d, t)
    try:
        u = UHFWalkers([a.copy(), b.copy()]).orthonormalize()
        r, norms = RHFWalkers(a.copy()).orthogonalize()
        got = [x.cpu().numpy() for x in (u.data[0], u.data[1], r.data, norms)]
    finally:
        for d in keys:
            _lib.set_tuning(d, None)
    assert rel_err(got[0], qs[0]) < _tol(a)
    assert rel_err(got[1], qs[1]) < _tol(b)
    assert rel_err(got[2], qa) < _tol(a)
    # ratios: the squares of 64 columns' norms overflow in the comparison itself
    assert rel_err(got[3] / na**2, np.ones(W)) < 100 * nelec[0] * np.finfo(float).eps * 10


@pytest.mark.parametrize("norb,no", [(7, 6), (40, 9), (300, 59)])
def test_qr_of_a_triangular_matrix(norb, no):
    """Zero reflectors: real upper triangular walkers come back as the identity's columns."""
    from ad_afqmc_b200.walkers import RHFWalkers

    rng = np.random.default_rng(1)
    a = np.zeros((3, norb, no), complex)
    a[:, :no] = np.triu(rng.standard_normal((3, no, no))) + 3.0 * np.eye(no)
    q_ref, _ = orc.qr_restricted(a)
    q = RHFWalkers(a.copy()).orthonormalize().data.cpu().numpy()
    assert rel_err(q, q_ref) < _tol(a[:, :no])
