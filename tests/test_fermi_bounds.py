"""The error bound of the Fermi search's FP32 passes against the float sums that they take, restated on
the CPU: a thread adds the terms of its slice one after another in FP32, and the search may take a level as
above or below the electron count only where the sum is off by more than the bound."""
import numpy as np
import pytest


def _bound(terms, beta=0.0, span=0.0):
    return 1e-4 + 4e-7 * beta * span + 6e-8 * terms


@pytest.mark.parametrize("terms", [68, 1700, 30000, 400000])
def test_float_sum_within_the_bound(terms):
    """Terms whose roundings all go the same way, the worst order there is."""
    worst = 0.0
    for v in (1.0 + 2.0 ** -23, 1.0 / 3.0, 0.7000001, 1.0 - 2.0 ** -24, 0.1):
        t = np.float32(v)
        s = np.add.accumulate(np.full(terms, t, dtype=np.float32))[-1]
        worst = max(worst, abs(float(s) / (terms * float(t)) - 1.0))
    assert worst < _bound(terms)
    if terms >= 30000:  # without the term for the sum's length the bound is too small
        assert worst > 1e-4


def test_source_has_the_bound():
    import os
    import sqminiapp_gb300
    src = open(os.path.join(os.path.dirname(sqminiapp_gb300.__file__), "csrc", "fermi.cu")).read()
    assert "1e-4 + 4e-7 * beta * span + 6e-8 * (double)((n + stride - 1) / stride)" in src
