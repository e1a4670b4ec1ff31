"""Log-Gaussian broadening where bins far from the output frequency are left out: widths that leave
out nearly all bins, some, and none, against the oracle.

A term's x = ln(w / E) / b (x^2 <= 745) carries the rounding of the ratio, eps / b, and those of the
logarithm and the division, 4 eps |x| at most; exp(-x^2) turns an error d of x into 2 |x| d, on either
side; the terms are positive."""
import numpy as np
import pytest

from nrg_b200 import Context
from oracle import nrg_oracle as O

pytestmark = pytest.mark.gpu


def _rtol(b):
    return 2 * (2 * 27.5 / b + 8 * 746) * np.finfo(float).eps


@pytest.mark.parametrize("b", [1e-3, 0.05, 0.6, 4.0, 40.0])
@pytest.mark.parametrize("nbin", [1, 255, 256, 4001])
def test_left_out_bins_add_nothing(b, nbin):
    rng = np.random.default_rng(nbin)
    bins = np.zeros((2 * nbin, 2), order="F")
    bins[:, 0] = np.tile(10.0 ** np.linspace(-18.0, 12.0, nbin), 2)
    bins[nbin:, 0] *= -1.0
    bins[:, 1] = rng.random(2 * nbin) * (rng.random(2 * nbin) < 0.9)
    w = np.concatenate([10.0 ** np.linspace(-18.0, 12.0, 61), -(10.0 ** np.linspace(-18.0, 12.0, 31))])
    with Context(0) as ctx:
        A = ctx.broaden_log_gaussian(bins, nbin, 2, b, w)
    R = O.broaden_log_gaussian(bins, nbin, 2, b, w)
    assert np.all(np.abs(A - R) <= _rtol(b) * np.abs(R) + 1e-290)
