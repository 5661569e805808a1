"""Solves of several sizes launched from several threads at once.

Each thread has its own engine and stream; together they launch the same kernels with different
amounts of shared memory.  Every launch succeeds, and energies, overlaps, steps and QR are the
bits that the solve gives alone."""

import threading

import pytest
import torch

from ad_afqmc_b200.synthetic import make_system
from tests._helpers import device_system

pytestmark = pytest.mark.gpu

SIZES = [(24, 3, 30), (70, 40, 20), (50, 11, 40), (64, 20, 25)]


def _solve(norb, no, nchol, precision):
    from ad_afqmc_b200.walkers import RHFWalkers

    W = 6
    sys_ = make_system(norb, (no, no), nchol, seed=norb, trial="rhf", chol_scale=0.2)
    trial, ham, wave, prop, _ = device_system(sys_, "restricted", 0.005, W, precision=precision)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(no)
    mo = torch.as_tensor(sys_.mo_coeff, device="cuda")
    w0 = mo + 0.05 * torch.randn(W, norb, no, dtype=torch.complex128, device="cuda", generator=gen)
    fields = torch.randn(W, nchol, dtype=torch.float64, device="cuda", generator=gen)
    eng = prop.engine(ham, trial, wave)

    def once():
        pd = prop.init_prop_data(trial, wave, dict(ham, e_estimate=0.0), 0, init_walkers=RHFWalkers(w0.clone()))
        e = trial.calc_energy(pd["walkers"], ham, wave, engine=eng)
        pd = prop.propagate_constrained(trial, ham, pd, fields, wave)
        q = pd["walkers"].orthonormalize()
        return [e, trial.calc_overlap(q, wave), q.data.clone(), pd["weights"].clone()]

    return once


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_threads(precision):
    solves = [_solve(*s, precision) for s in SIZES]
    alone = [s() for s in solves]
    torch.cuda.synchronize()
    failed = []

    def work(i):
        try:
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                for _ in range(60):
                    got = solves[i]()
                stream.synchronize()
            if not all(torch.equal(a, b) for a, b in zip(got, alone[i])):
                failed.append((i, "bits"))
        except Exception as e:  # noqa: BLE001 - reported below
            failed.append((i, repr(e)))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(solves))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed


def test_scratch_per_stream():
    """Overlaps, Green's functions and QR on two streams do not share scratch."""
    from ad_afqmc_b200._engine import small_work

    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(a):
        x = small_work(6)
        again = small_work(6)
    with torch.cuda.stream(b):
        y = small_work(6)
    assert x.data_ptr() == again.data_ptr() != y.data_ptr()
