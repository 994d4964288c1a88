"""Which route an FP32 match takes, by the scratch it asks for, and the same choice on
both sides of each line."""

import numpy as np
import pytest

from custom_madi_gb300 import _native as N


def _need(n_vox, n_lib, F):
    return int(N.lib().madi_match_scratch_bytes(n_vox, n_lib, F, N.MADI_MATCH_FP32, 32))


def test_fp32_routes_by_size():
    """One part up to two chunks of 128 entries, parts (8 bytes a voxel) beyond, the
    index from 4e9 voxel x entry x feature products on, 4,096 voxels and 1,024 entries."""
    for n_vox, n_lib, F in ((1, 1, 1), (50, 200, 5), (50, 256, 20), (400_000, 256, 20)):
        assert _need(n_vox, n_lib, F) == 256
    for n_vox, n_lib, F in ((50, 257, 5), (9_999, 20_000, 20), (4_095, 1_000_000, 32), (1_000, 1_023, 32)):
        assert _need(n_vox, n_lib, F) == 256 + 8 * n_vox
    for n_vox, n_lib, F in ((10_000, 20_000, 20), (4_096, 40_000, 32), (200_000, 1_024, 20)):
        assert _need(n_vox, n_lib, F) > 256 + 8 * n_vox


@pytest.mark.gpu
@pytest.mark.parametrize("free", (False, True))
@pytest.mark.parametrize("n_vox, n_lib, F", [(50, 256, 20), (50, 257, 20), (9_999, 20_000, 20), (10_000, 20_000, 20),
                                             (155_520, 300, 7), (155_648, 300, 7), (4_096, 40_000, 32)])
def test_both_sides_of_each_line_choose_alike(n_vox, n_lib, F, free):
    from test_gpu_match_routes import _data, _match
    vox, lib = _data("decays", n_vox, n_lib, F, np.random.default_rng(n_vox))
    need, a = _match(vox, lib, free)
    assert need == _need(n_vox, n_lib, F)
    _, b = _match(vox, lib, free, scratch_bytes=256)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
    score = -2.0 * vox.astype(np.float64) @ lib.T.astype(np.float64)        # fp64, to fp32 rounding of the chosen score
    if free:
        score = -np.maximum(-0.5 * score, 0.0) ** 2 / (lib.astype(np.float64) ** 2).sum(1)
    else:
        score += (lib.astype(np.float64) ** 2).sum(1)
    best = score.min(axis=1)
    got = score[np.arange(n_vox), a[0]]
    assert (got - best <= 64 * 2.0 ** -24 * ((vox.astype(np.float64) ** 2).sum(1) + (lib.astype(np.float64) ** 2).sum(1).max())).all()
