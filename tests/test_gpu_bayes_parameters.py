"""Parameters of the Bayesian fit that agree in most of their bits, and parameters
outside fp32's range: the fit uses all 53 bits of each."""

import numpy as np
import pytest

from test_gpu_bayes_routes import _fit

pytestmark = pytest.mark.gpu


def _flat(n_vox, n_lib, F, par, free, small):
    """Every entry has the same signal and weight, so every posterior is uniform over the entries."""
    rng = np.random.default_rng(3)
    lib = np.tile(np.exp(-np.linspace(0.0, 2.0, F)), (n_lib, 1)).astype(np.float32)
    vox = (lib[:1] + 0.02 * rng.standard_normal((n_vox, F))).astype(np.float32)
    return _fit(vox, lib, par, np.zeros(n_lib), free, 0.02, small)[1]


@pytest.mark.parametrize("free", (False, True))
@pytest.mark.parametrize("small", (False, True))
@pytest.mark.parametrize("n_vox, n_lib, F", [(100, 300, 5), (500, 1_100, 20), (20_000, 300, 28)])
def test_parameters_that_nearly_agree(n_vox, n_lib, F, small, free):
    """Means and standard deviations of parameters whose spread is 2^-50 to 2^-20 of their size.

    Sums of n exact weights 1: the fp32 difference rounds by 2^-24, the compensated
    sums of d and d^2 by a few 2^-24 of the largest term."""
    rng = np.random.default_rng(n_lib)
    k = rng.permutation(n_lib).astype(np.float64)
    par = np.stack([1.7 + k * 2.0 ** -51, 3.0e6 * (1.0 + k * 2.0 ** -40), 0.011 * (1.0 + k * 2.0 ** -30)], axis=1)
    out = _flat(n_vox, n_lib, F, par, free, small)
    for i in range(3):
        std = par[:, i].std()
        mean = np.mean(par[:, i] - par[0, i]) + par[0, i]
        assert np.abs(out[i] - mean).max() <= 1e-5 * std + np.spacing(mean)
        assert np.abs(out[3 + i] - std).max() <= 1e-5 * std


@pytest.mark.parametrize("scale", (3e38, 1e39, 1e120, 1e-30, 1e-36, 1e-120))
def test_parameters_outside_fp32(scale):
    """Parameters far beyond fp32's range whose differences lie in it keep their mean
    (the differences are taken in fp64)."""
    k = np.arange(200.0)
    step = min(1e30, scale) if scale > 1.0 else max(1e-36, scale * 1e-3)
    par = np.stack([scale + k * step, np.full(200, 4e3), scale + k[::-1] * step], axis=1)
    out = _flat(64, 200, 8, par, False, True)
    out2 = _flat(700, 1_200, 8, np.tile(par, (6, 1)), False, False)
    for o in (out, out2):
        for i in (0, 2):
            want = np.mean(par[:, i] - par[0, i]) + par[0, i]
            assert np.allclose(o[i], want, rtol=1e-6, atol=0.0)
        assert np.allclose(o[1], 4e3, rtol=1e-12)
