"""FP32 match against libraries of more than 2^30 entries."""

import pytest

from custom_madi_gb300 import _native as N


@pytest.mark.parametrize("n_lib", (1_500_000_000, 2_000_000_000, 2 ** 31 - 1))
def test_route_of_a_very_large_library(n_lib):
    """No index (its counts are 32 bits); small fits split the library."""
    need = N.lib().madi_match_scratch_bytes
    assert need(100, n_lib, 1, N.MADI_MATCH_FP32, 32) == 256 + 8 * 100
    assert need(4_096, n_lib, 1, N.MADI_MATCH_FP32, 32) == 256 + 8 * 4_096
    assert N.lib().madi_bayes_work_bytes(100, n_lib, 1) == 256


@pytest.mark.gpu
def test_match_of_one_and_a_half_billion_entries():
    """One feature (6 GB): the entry nearest to each voxel, lowest index of equals, from
    the first and the last parts of the library."""
    import torch
    from custom_madi_gb300.fitters_gpu import match_device
    n_lib = 1_500_000_000
    lib = torch.zeros((n_lib, 1), device="cuda")
    spots = [0, 127, 128, n_lib // 2, n_lib - 129, n_lib - 128, n_lib - 1]
    for k, j in enumerate(spots):
        lib[j] = 1.0 + k
    lib[n_lib - 5] = 1.0 + 3                      # an equal of spots[3], later
    vox = torch.tensor([[1.0 + k] for k in range(len(spots))] + [[0.0]], device="cuda")
    idx, resid, _ = match_device(vox, lib)
    assert idx.cpu().tolist() == spots + [1]
    assert bool((resid == 0.0).all())
    del lib
    torch.cuda.empty_cache()
