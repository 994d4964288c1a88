"""The FP32 match where squares leave fp32's range."""

import numpy as np
import pytest

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
