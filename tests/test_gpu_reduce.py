"""madi_reduce_Y against a plain fp64 numpy reduction: run and column-block edges,
walker remainders, phases beyond the fixed-point range.

A term's cos / sin is good to 2e-12 (products rounded to 2^-40, phase to 2^-44
turn); numpy's own phase rounds at |phase| 2^-53, and the fp64 path's too."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(n_walkers, n_cols, n_grid, scale, per_run, seed):
    rng = np.random.default_rng(seed)
    Y = np.cumsum(rng.normal(0.0, 1.0, (n_walkers, n_grid, 3)), axis=1)
    runs = (n_cols + per_run - 1) // per_run
    trip = np.repeat(rng.integers(0, n_grid, (runs, 3)), per_run, axis=0)[:n_cols].astype(np.int32)
    return Y, trip, rng.uniform(0.0, scale, n_cols)


@pytest.mark.parametrize("n_walkers, n_cols, n_grid, scale, per_run", [
    (1, 1, 2, 1.0, 1),             # smallest
    (33, 25, 129, 0.5, 25),        # one run
    (64, 255, 47, 2.0, 7),         # a column short of a warp row
    (37, 257, 47, 2.0, 1),         # every column its own run
    (65, 512, 47, 2.0, 25),        # the last width of the 256-thread form
    (65, 513, 47, 2.0, 25),        # the first of the 512-thread form
    (130, 1024, 129, 0.3, 25),     # a full column block, runs across thread rows
    (40, 1025, 512, 0.3, 1),       # 1,024 runs in a block (one walker's dM at a time), one column over
    (70, 600, 129, 40.0, 25),      # phases beyond 127 turns: some chunks in fp64
    (700, 2100, 129, 0.4, 25),     # several walker blocks, ragged
])
def test_reduce_Y_matches_fp64(n_walkers, n_cols, n_grid, scale, per_run):
    import torch
    from custom_madi_gb300 import _native as N
    Y, trip, coef = _case(n_walkers, n_cols, n_grid, scale, per_run, seed=n_cols)
    dm = (Y[:, trip[:, 0]] + Y[:, trip[:, 1]]) - Y[:, trip[:, 2]]          # [walkers, cols, 3]
    ph = coef[None, :, None] * dm
    tol = 3 * n_walkers * (2e-12 + 4.0 * 2.0 ** -53 * np.abs(ph).max())
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (Y, trip[:, 0], trip[:, 1], trip[:, 2], coef)]
    out = []
    for _ in range(2):
        cs, sn = torch.empty_like(dev[4]), torch.empty_like(dev[4])
        N.reduce_Y(dev[0], n_walkers, n_grid, *dev[1:], cs, sn, torch.cuda.current_stream())
        out.append((cs.cpu().numpy(), sn.cpu().numpy()))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
    assert np.abs(out[0][0] - np.cos(ph).sum(axis=(0, 2))).max() <= tol
    assert np.abs(out[0][1] - np.sin(ph).sum(axis=(0, 2))).max() <= tol
