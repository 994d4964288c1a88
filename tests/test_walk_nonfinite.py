"""Steps that are not finite, or not in fp32: as a walk's sigma they are refused; in a
replay stream they end that walker's walk or leave it without a position, and do
nothing to the walkers beside it."""

import ctypes as C

import numpy as np
import pytest

from custom_madi_gb300 import _native as N
from custom_madi_gb300.config import SimConfig


@pytest.mark.parametrize("precision, sigma", [(32, np.nan), (32, np.inf), (32, -np.inf), (32, 1e39), (64, np.nan), (64, np.inf)])
def test_sigma_that_is_not_finite_is_refused(precision, sigma):
    """Before anything is launched: no device is needed."""
    word = C.create_string_buffer(4096)
    d = N.MadiWalkDesc()
    d.geoms = d.jobs = d.accum = d.occupancy = d.counters = d.Y = d.inside_trace = d.work_counter = C.addressof(word)
    d.n_geoms = d.n_jobs = d.n_tiles = 1
    d.tile_walkers, d.precision, d.rng, d.out_mode = 128, precision, N.MADI_RNG_PHILOX, N.MADI_OUT_Y
    d.n_steps, d.steps_per_h, d.n_grid = 1, 1, 2
    d.sigma = sigma
    with pytest.raises(ValueError, match="sigma"):
        N.check(N.lib().madi_walk(C.byref(d), None), "madi_walk")


@pytest.mark.gpu
@pytest.mark.parametrize("precision", (32, 64))
@pytest.mark.parametrize("mode, pp", [("periodic", 0.0), ("periodic", 0.3), ("si_fatal_escape", 0.0)])
def test_steps_that_are_not_finite(mode, pp, precision):
    """NaN, infinite and (fp32) overflowing steps of a stream: the walk ends, and up to
    such a step it equals the walk without the facet table, bit for bit (the label of
    a point that is nowhere depends on the cell the voxel rule looks at first)."""
    import torch
    from custom_madi_gb300.ensemble import create_ensemble
    from custom_madi_gb300.walker_gpu import WalkBatch, WalkJob, WalkRandomStream, make_walk_random_stream
    n = 225
    over = dict(boundary_mode="periodic", n_cells=27) if mode == "periodic" else {}
    cfg = SimConfig(n_walkers=n, n_ensembles=1, ts=0.01, T_max_ms=3.0, h_ms=0.1, small_deltas=[1.0], big_deltas=[2.0],
                    b_values=[0.0, 1000.0], **over)
    ens = create_ensemble(2.0e5, 4.0, cfg, seed=5, verify_vi=False, measure_vi=False)
    s = make_walk_random_stream(cfg, 3, ens)
    inc, u = s.increments.copy(), s.acceptance_uniforms.copy()
    bad = [np.nan, np.inf, -np.inf, 1e39, -1e39]
    for k in range(60):                      # one axis or all three, at early and late steps
        w, step = 3 * k, 1 + 4 * k
        inc[step, w, (k % 4 if k % 4 < 3 else slice(None))] = bad[k % len(bad)]
        u[step, w] = 0.999 if k % 2 else 0.0
    stream = WalkRandomStream(s.initial_positions, inc, u)
    out = []
    for table in (True, False):
        ens._device.clear()
        dev = ens.device()
        if not table:
            dev.struct.n_cells = 0
        b = WalkBatch([WalkJob(ens, pp, 11, n)], cfg, out_mode=N.MADI_OUT_Y, stream=stream, precision=precision)
        b.launch()
        torch.cuda.synchronize()
        out.append((b.Y.cpu().numpy(), b.inside_trace.cpu().numpy(), b.counters_np()[0]))
    ens._device.clear()
    (Y, inside, cnt), (Yv, inside_v, cnt_v) = out
    assert cnt[0] == cnt_v[0] == n and cnt[1] + cnt[2] > 0
    assert precision == 64 or cnt[8] > 0                     # facet passes were made
    last = np.full(n, cfg.n_grid)
    for k in range(60):
        last[3 * k] = (1 + 4 * k) // cfg.steps_per_h          # storage points at or before the step
    for w in range(n):
        assert np.isfinite(Y[w, :last[w]]).all()
        assert np.array_equal(Y[w, :last[w]], Yv[w, :last[w]]) and np.array_equal(inside[w, :last[w]], inside_v[w, :last[w]])
