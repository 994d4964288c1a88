"""Launches too small for the GPU take more of it only where they have it to
themselves: by the caller's word, or as the only walk being waited for."""

import threading

import numpy as np
import pytest

from custom_madi_gb300 import walker_gpu as W
from custom_madi_gb300.config import SimConfig


def test_walk_in_flight_counts():
    """The only walk is told so; nested, in another thread and after an error the count is right."""
    seen = {}

    def other():
        with W.walk_in_flight() as only:
            seen["beside"] = only
    with W.walk_in_flight() as only:
        assert only
        t = threading.Thread(target=other)
        t.start()
        t.join()
        with W.walk_in_flight() as again:
            assert not again
    assert seen == {"beside": False}
    with pytest.raises(RuntimeError, match="x"):
        with W.walk_in_flight() as only:
            assert only
            raise RuntimeError("x")
    with W.walk_in_flight() as only:
        assert only


def test_default_launch_makes_no_promise():
    assert W.LaunchConfig().alone is False
    lc = W.LaunchConfig(tile_walkers=64, persistent=False)
    assert W._launch_alone(lc, True) == W.LaunchConfig(tile_walkers=64, persistent=False, alone=True)
    assert W._launch_alone(lc, False) == lc and W._launch_alone(None, False) == W.LaunchConfig()


def _pgse(n):
    from custom_madi_gb300 import signal as S
    from custom_madi_gb300 import workloads as WL
    cfg = WL.plain_config(n_walkers=n, directions=24)
    c = S.build_columns(cfg)
    return cfg, W.pair_layout(c.j_delta, c.j_Delta, c.j_sum, c.phase_coef)


@pytest.mark.gpu
@pytest.mark.parametrize("n", (10_000, 20_000))
def test_overlapping_small_launches_share_the_gpu(n):
    """Two small launches on two streams, neither promised the GPU, run side by side:
    well under the time of one after the other (they used to take 1.9x one's time)."""
    import torch
    from custom_madi_gb300.ensemble import create_ensemble
    cfg, lay = _pgse(n)
    ens = create_ensemble(2.0e5, 4.0, cfg, seed=3, verify_vi=False, measure_vi=False)
    batches = [W.WalkBatch([W.WalkJob(ens, 0.01, 17 + i, n)], cfg, layout=lay, dirs=cfg.direction_array()) for i in range(2)]
    streams = [torch.cuda.Stream() for _ in batches]

    def time(k):
        ms = []
        for _ in range(6):
            torch.cuda.synchronize()
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            for batch, s in list(zip(batches, streams))[:k]:
                s.wait_stream(torch.cuda.current_stream())
                batch.launch(s)
            for s in streams[:k]:
                torch.cuda.current_stream().wait_stream(s)
            b.record()
            torch.cuda.synchronize()
            ms.append(a.elapsed_time(b))
        return float(np.median(ms[1:]))
    assert time(2) < 1.5 * time(1)


@pytest.mark.gpu
@pytest.mark.parametrize("n, tile, out", [
    (1, 32, "fused"), (33, 32, "fused"), (700, 64, "fused"), (225, 128, "fused"), (9_999, 128, "fused"),
    (14_592, 128, "fused"), (14_721, 128, "fused"), (300, 256, "fused"), (225, 128, "Y"), (5_003, 128, "Y"),
])
@pytest.mark.parametrize("persistent", [True, False])
def test_a_launch_that_is_alone_walks_the_same(n, tile, out, persistent):
    """Sums, occupancy, stored Y and counters with the promise equal those without, bit for bit."""
    import torch
    from custom_madi_gb300 import _native as N
    from custom_madi_gb300 import signal as S
    from custom_madi_gb300.ensemble import create_ensemble
    fused = out == "fused"
    over = dict(boundary_mode="periodic", n_cells=40) if fused else {}
    cfg = SimConfig(n_walkers=n, n_ensembles=1, ts=0.01, T_max_ms=3.1, h_ms=0.31, small_deltas=[0.31], big_deltas=[1.55],
                    b_values=[0.0, 1000.0, 3000.0], **over)
    ens = create_ensemble(2.0e5, 3.0, cfg, seed=3, verify_vi=False, measure_vi=False)
    c = S.build_columns(cfg)
    lay = W.pair_layout(c.j_delta, c.j_Delta, c.j_sum, c.phase_coef) if fused else None
    res = []
    for alone in (True, False):
        b = W.WalkBatch([W.WalkJob(ens, 0.05, 11, n, walker_base=5)], cfg, layout=lay,
                        out_mode=N.MADI_OUT_FUSED if fused else N.MADI_OUT_Y,
                        launch=W.LaunchConfig(tile_walkers=tile, persistent=persistent, alone=alone))
        b.launch()
        torch.cuda.synchronize()
        res.append([x.cpu().numpy() for x in (b.occupancy, b.counters, b.accum if fused else b.Y)])
        assert res[-1][1][0, 0] == n
    for x, y in zip(*res):
        assert np.array_equal(x, y)


@pytest.mark.gpu
def test_small_walks_from_several_threads():
    """Threads that each wait for small walks of their own get the sums of a walk by itself."""
    from custom_madi_gb300 import signal as S
    from custom_madi_gb300.ensemble import create_ensemble
    cfg, _ = _pgse(3_000)
    c = S.build_columns(cfg)
    cols = (c.j_delta, c.j_Delta, c.j_sum, c.phase_coef)
    ens = create_ensemble(2.0e5, 4.0, cfg, seed=3, verify_vi=False, measure_vi=False)
    ens.device()
    ref = [W.simulate_jobs([W.WalkJob(ens, 0.01, 17 + i, 3_000)], cfg, cols)[0] for i in range(4)]
    got, errors = [None] * 4, []

    def work(i):
        import torch
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(3):
                    got[i] = W.simulate_jobs([W.WalkJob(ens, 0.01, 17 + i, 3_000)], cfg, cols)[0]
        except Exception as e:           # reported by the assertion below
            errors.append(e)
    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for a, b in zip(ref, got):
        assert np.array_equal(a["cos_fixed"], b["cos_fixed"]) and np.array_equal(a["sin_fixed"], b["sin_fixed"])
        assert np.array_equal(a["occupancy"], b["occupancy"]) and a["counters"] == b["counters"]
