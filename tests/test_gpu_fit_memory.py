"""FP32 fits where there is no room for the search index: accepted as before it, same results."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _inputs(n_vox=20_000, n_lib=12_000, F=20):
    rng = np.random.default_rng(2)
    t = np.sort(rng.uniform(0.0, 3.0, F))
    lib = 0.6 * np.exp(-t * rng.uniform(0.1, 3.0, (n_lib, 1))) + 0.4 * np.exp(-t * rng.uniform(0.1, 1.0, (n_lib, 1)))
    vox = lib[rng.integers(0, n_lib, n_vox)] + 0.03 * rng.standard_normal((n_vox, F))
    return vox.astype(np.float32), lib.astype(np.float32)


@pytest.mark.parametrize("free", (False, True))
def test_server_budget_that_holds_the_fit_but_not_the_index(free):
    """A budget of the voxels, the results and the column means, which such a request
    needed before there was an index, still admits it."""
    from custom_madi_gb300 import workloads as WL
    from custom_madi_gb300 import signal as S
    from custom_madi_gb300.fitters_gpu import match_device
    from custom_madi_gb300.serving import FitRequest, Server
    from custom_madi_gb300.walker_gpu import pair_layout
    vox, lib = _inputs()
    n, f = vox.shape
    cfg = WL.plain_config(n_walkers=1_000, directions=6)
    c = S.build_columns(cfg)
    lay = pair_layout(c.j_delta, c.j_Delta, c.j_sum, c.phase_coef)
    fit = n * f * 4 + n * 12 + 256 + 512
    pool = Server(cfg, lay, cfg.direction_array(), library=lib, n_slots=1).pool_bytes
    srv = Server(cfg, lay, cfg.direction_array(), library=lib, n_slots=1, budget_bytes=fit + pool)
    rec = srv.run([FitRequest(vox, precision="fp32", free_s0=free)], realtime=False)["records"][0]
    ref = match_device(vox, lib, free_s0=free)
    assert rec.nbytes == fit
    assert np.array_equal(rec.result["best_idx"], ref[0].cpu().numpy())
    assert np.array_equal(rec.result["best_resid"], ref[1].cpu().numpy())
    with pytest.raises(ValueError, match="budget"):
        Server(cfg, lay, cfg.direction_array(), library=lib, n_slots=1, budget_bytes=fit + pool - 1).run(
            [FitRequest(vox, precision="fp32", free_s0=free)], realtime=False)


@pytest.mark.parametrize("free", (False, True))
def test_a_device_without_room_for_the_index(free, monkeypatch):
    """The allocation of the large scratch fails (on the host side of the allocator)."""
    import torch
    from custom_madi_gb300 import fitters_gpu as G
    vox, lib = _inputs()
    par = np.random.default_rng(4).uniform(1.0, 2.0, (3, len(lib)))
    q = np.ones(len(lib))
    ref = G.match_device(vox, lib, free_s0=free)
    fit = G.bayes_fit_gpu(vox[:2_000], lib, *par, 0.02, fit_s0=free, quadrature_weights=q)
    empty, refused = torch.empty, []

    def no_room(*a, **kw):
        if kw.get("dtype") == torch.uint8 and a[0] > 1024:
            refused.append(a[0])
            raise torch.cuda.OutOfMemoryError("CUDA out of memory")
        return empty(*a, **kw)
    monkeypatch.setattr(torch, "empty", no_room)
    got = G.match_device(vox, lib, free_s0=free)
    got_fit = G.bayes_fit_gpu(vox[:2_000], lib, *par, 0.02, fit_s0=free, quadrature_weights=q)
    with pytest.raises(torch.cuda.OutOfMemoryError):
        G.match_device(vox, lib, precision="bf16")
    assert len(refused) == 3
    for x, y in zip(ref, got):
        assert x is y is None or torch.equal(x, y)
    for k in fit:
        assert np.array_equal(fit[k], got_fit[k])
