"""Prepared buffer and workspace together take no more than these sizes.

The bounds are what they took with operand rows of multiples of eight values and FP64
buffers in every precision; rows of 64 values must not make a solve larger."""

import pytest

from ad_afqmc_b200 import _lib

# norb, no, nchol, walkers: (restricted, unrestricted) bytes for fp64, mixed, mixed_hi
BOUNDS = {
    (33, 8, 132, 64): [5003776, 6469376, 7612928, 9691392, 8849920, 11234816],
    (65, 13, 260, 200): [46428160, 58551552, 70124032, 86976256, 81295872, 100512512],
    (97, 24, 480, 231): [161601536, 201152768, 238740480, 296509184, 275158784, 342036224],
    (157, 39, 863, 231): [522503168, 662742272, 778803456, 984651776, 901295872, 1139948800],
    (200, 40, 1000, 512): [1269934080, 1553489408, 1891406336, 2304657920, 2185758464, 2663858176],
    (300, 60, 1500, 1024): [4939075072, 6057753856, 7482079232, 9115440896, 8679853312, 10570556416],
}


@pytest.mark.parametrize("shape", BOUNDS, ids=lambda s: f"n{s[0]}")
def test_footprint(shape):
    norb, no, nchol, W = shape
    types = [(_lib.AFQ_RESTRICTED, _lib.AFQ_TRIAL_RHF), (_lib.AFQ_UNRESTRICTED, _lib.AFQ_TRIAL_UHF)]
    got = [sum(_lib.sizes(_lib.make_dims(norb, (no, no), nchol, W, wt, tt, 6, precision, 0.005)))
           for precision in (0, 1, 2) for wt, tt in types]
    assert all(g <= b for g, b in zip(got, BOUNDS[shape])), got
