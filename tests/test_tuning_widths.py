"""Records may name the exchange column widths that are compiled, and no others."""

import pytest

from ad_afqmc_b200 import _lib


def _dims(no, precision):
    return _lib.make_dims(70, (no, no), 90, 3, _lib.AFQ_RESTRICTED, _lib.AFQ_TRIAL_RHF, 6, precision, 0.005)


@pytest.mark.parametrize("precision", [1, 2])
@pytest.mark.parametrize("bn", [16, 48, 72, 100, 112, 127, 144, 160, 256, -64])
def test_other_widths_are_refused(bn, precision):
    d = _dims(5, precision)
    with pytest.raises(_lib.AfqError):
        _lib.set_tuning(d, _lib.afq_tuning.from_dict({"exch_bn": bn}))
    assert _lib.get_tuning(d).as_dict()["exch_bn"] == 80


@pytest.mark.parametrize("bn", [32, 64, 80, 96, 128])
def test_compiled_widths_are_taken(bn):
    d = _dims(5, 1)
    try:
        _lib.set_tuning(d, _lib.afq_tuning.from_dict({"exch_bn": bn}))
        assert _lib.get_tuning(d).as_dict()["exch_bn"] == bn
    finally:
        _lib.set_tuning(d, None)
