"""The FP32 match and the Bayesian fit where squares leave fp32's range."""

import numpy as np
import pytest

from test_gpu_bayes_routes import _fit
from test_gpu_match_routes import _match

pytestmark = pytest.mark.gpu


def _decays(rng, n_vox, n_lib, F):
    t = np.sort(rng.uniform(0.0, 3.0, F))
    lib = 0.6 * np.exp(-t * rng.uniform(0.1, 3.0, (n_lib, 1))) + 0.4 * np.exp(-t * rng.uniform(0.1, 1.0, (n_lib, 1)))
    return lib[rng.integers(0, n_lib, n_vox)] + 0.03 * rng.standard_normal((n_vox, F)), lib


@pytest.mark.parametrize("n_vox, n_lib, F", [(3, 200, 5), (3_001, 5_000, 12), (20_000, 12_000, 20)])   # plain, split, indexed
@pytest.mark.parametrize("small", (False, True))
def test_free_s0_entry_whose_norm_overflows(n_vox, n_lib, F, small):
    """The score -(m.r)^2 / |r|^2 of an entry whose |r|^2 overflows is -0: it is taken
    where no other entry has m.r > 0."""
    rng = np.random.default_rng(n_vox)
    vox, lib = _decays(rng, n_vox, n_lib, F)
    vox, lib = np.abs(vox) * 1e-3, -np.abs(lib)
    lib[[17, 150]] = 2e19
    _, (idx, resid, s0) = _match(vox.astype(np.float32), lib.astype(np.float32), True, scratch_bytes=256 if small else None)
    assert (idx == 17).all() and (s0 == 0.0).all()


@pytest.mark.parametrize("free", (False, True))
@pytest.mark.parametrize("scale_vox, scale_lib", [(1e-20, 1e-20), (1e-21, 1e-21), (1e-22, 1e-22), (1.0, 1e-22), (1e3, 1e-23)])
def test_indexed_match_of_subnormal_squares_equals_scan(scale_vox, scale_lib, free):
    n_vox, n_lib, F = 20_000, 12_000, 20
    vox, lib = _decays(np.random.default_rng(7), n_vox, n_lib, F)
    vox, lib = (vox * scale_vox).astype(np.float32), (lib * scale_lib).astype(np.float32)
    lib[::3] *= -1.0                                     # free S0: not every entry has m.r > 0
    need, a = _match(vox, lib, free)
    assert need > 256 + 8 * n_vox                        # the index
    _, b = _match(vox, lib, free, scratch_bytes=256)
    for x, y in zip(a, b):
        assert np.array_equal(x, y, equal_nan=True)


@pytest.mark.parametrize("scale, sigma", [(1e-21, 1e-19), (1e-18, 5e-20), (1e-16, 1e-18)])
def test_indexed_fit_of_subnormal_squares_equals_plain(scale, sigma):
    rng = np.random.default_rng(8)
    vox, lib = _decays(rng, 3_000, 2_000, 20)
    par = np.exp(rng.uniform(np.log([1.0, 4e3, 0.01]), np.log([130.0, 5e7, 200.0]), (len(lib), 3)))
    logq = np.log(rng.uniform(0.2, 1.2, len(lib)))
    args = ((vox * scale).astype(np.float32), (lib * scale).astype(np.float32), par, logq, False, sigma)
    need, a = _fit(*args, small=False)
    assert need > 256
    _, b = _fit(*args, small=True)
    assert np.array_equal(a, b, equal_nan=True)
