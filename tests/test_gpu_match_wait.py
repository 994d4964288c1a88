"""A bounded wait of the indexed FP32 match that runs out is reported."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("free", (False, True))
@pytest.mark.parametrize("n_vox, n_lib", [(20_000, 12_000), (130_000, 2_000), (300_000, 1_024)])   # 4, 2, 1 warps a group
def test_fp32_bounded_wait_timeout_is_reported(n_vox, n_lib, free):
    """madi_match_wait returns MADI_ERR_TIMEOUT, the voxels have index -1 and NaN
    instead of what was in memory, and the next call on the same stream is whole.  The
    wait is made to run out by the test-only flag (a barrier nothing completes)."""
    import torch
    from custom_madi_gb300 import _native as N
    from custom_madi_gb300.fitters_gpu import match_device
    rng = np.random.default_rng(n_lib)
    t = np.sort(rng.uniform(0.0, 3.0, 20))
    lib = 0.6 * np.exp(-t * rng.uniform(0.1, 3.0, (n_lib, 1))) + 0.4 * np.exp(-t * rng.uniform(0.1, 1.0, (n_lib, 1)))
    vox = (lib[rng.integers(0, n_lib, n_vox)] + 0.03 * rng.standard_normal((n_vox, 20))).astype(np.float32)
    before = match_device(vox, lib, free_s0=free)
    out = match_device(vox, lib, free_s0=free, check=False, flags=N.MADI_MATCH_FLAG_TEST_STALL)
    with pytest.raises(N.MadiError, match="bounded wait ran out") as ei:
        out.check()
    assert ei.value.status == N.MADI_ERR_TIMEOUT and "were drained" in str(ei.value)
    assert bool((out[0] == -1).all()) and bool(torch.isnan(out[1]).all())
    assert not free or bool(torch.isnan(out[2]).all())
    good = match_device(vox, lib, free_s0=free)
    assert bool((good[0] >= 0).all())
    for x, y in zip(before, good):
        assert x is y is None or torch.equal(x, y)
