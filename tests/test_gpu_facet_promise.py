"""The walkers use the slot order and the annulus bound only where the geometry
promises them (MADI_FACETS_ORDERED)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", (32, 64))
@pytest.mark.parametrize("mode, n_cells", [("periodic", 27), ("si_fatal_escape", 0)])
def test_alpha_min_without_the_promise_is_not_read(mode, n_cells, precision, monkeypatch):
    """A geometry with its slots in descending order and any value in alpha_min, as a
    caller that knows neither may leave it, walks as the voxel-grid rule does."""
    import torch
    from custom_madi_gb300 import _native as N
    from custom_madi_gb300 import ensemble as E
    from custom_madi_gb300.config import SimConfig
    from custom_madi_gb300.walker_gpu import WalkBatch, WalkJob
    n = 2_000
    over = dict(boundary_mode="periodic", n_cells=n_cells) if mode == "periodic" else {}
    cfg = SimConfig(n_walkers=n, n_ensembles=1, ts=0.01, T_max_ms=4.0, small_deltas=[1.0], big_deltas=[2.0],
                    b_values=[0.0, 1000.0], **over)
    ens = E.create_ensemble(2.0e5, 2.6, cfg, seed=5, verify_vi=False, measure_vi=False)
    pack = E.pack_facets

    def descending(*a):
        stride, planes, nbr = pack(*a)
        return stride, np.ascontiguousarray(planes[:, ::-1]), np.ascontiguousarray(nbr[:, ::-1])
    monkeypatch.setattr(E, "pack_facets", descending)
    out = []
    for alpha_min in (7.0, 0.0, None):
        ens._device.clear()
        dev = ens.device()
        if alpha_min is None:
            dev.struct.n_cells = 0
        else:
            dev.struct.facet_stride = dev.facet_stride
            dev.struct.alpha_min = alpha_min
        b = WalkBatch([WalkJob(ens, 0.1, 11, n)], cfg, out_mode=N.MADI_OUT_Y, precision=precision)
        b.launch()
        torch.cuda.synchronize()
        cnt = b.counters_np()[0]
        out.append((b.Y.cpu().numpy(), b.inside_trace.cpu().numpy(), b.occupancy.cpu().numpy(), cnt[[0, 1, 2, 6, 7]]))
    ens._device.clear()
    for other in out[1:]:
        for x, y in zip(out[0], other):
            assert np.array_equal(x, y)
