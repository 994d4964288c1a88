"""Fits on a stream that is not the current one: ordered after the current stream's
work, their buffers kept until they are done."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SLEEP = 200_000_000                      # cycles of a pending kernel, ~0.1 s


def _inputs(n_vox, n_lib, F):
    rng = np.random.default_rng(n_vox)
    t = np.sort(rng.uniform(0.0, 3.0, F))
    lib = 0.6 * np.exp(-t * rng.uniform(0.1, 3.0, (n_lib, 1))) + 0.4 * np.exp(-t * rng.uniform(0.1, 1.0, (n_lib, 1)))
    vox = lib[rng.integers(0, n_lib, n_vox)] + 0.03 * rng.standard_normal((n_vox, F))
    par = np.exp(rng.uniform(np.log([1.0, 4e3, 0.01]), np.log([130.0, 5e7, 200.0]), (n_lib, 3)))
    return vox.astype(np.float32), lib.astype(np.float32), par, rng.uniform(0.2, 1.2, n_lib)


def _pending(vox, lib):
    """Device inputs that hold their values only after the current stream's pending work."""
    import torch
    M, L = torch.zeros(vox.shape, device="cuda"), torch.zeros(lib.shape, device="cuda")
    hv, hl = torch.from_numpy(vox).cuda(), torch.from_numpy(lib).cuda()
    torch.cuda.synchronize()
    torch.cuda._sleep(SLEEP)
    M.copy_(hv)
    L.copy_(hl)
    return M, L


@pytest.mark.parametrize("precision, free", [("fp32", False), ("fp32", True), ("bf16", False)])
@pytest.mark.parametrize("check", (True, False))
def test_match_on_a_side_stream(precision, free, check):
    import torch
    from custom_madi_gb300.fitters_gpu import match_device
    vox, lib, _, _ = _inputs(20_000, 12_000, 20)
    ref = [None if t is None else t.cpu() for t in match_device(vox, lib, free_s0=free, precision=precision)]
    side = torch.cuda.Stream()
    M, L = _pending(vox, lib)
    out = match_device(M, L, free_s0=free, precision=precision, stream=side, check=check)
    if not check:
        # the call's inputs and scratch are let go of while it waits, and their memory asked for again
        junk = [torch.full((1 << 20,), -1, dtype=torch.int32, device="cuda") for _ in range(16)]
        out.check()
        del junk
    for x, y in zip(ref, out):
        assert x is y is None or torch.equal(x, y.cpu())


@pytest.mark.parametrize("free", (False, True))
def test_bayes_on_a_side_stream(free):
    import torch
    from custom_madi_gb300.fitters_gpu import bayes_fit_gpu
    vox, lib, par, q = _inputs(5_000, 4_000, 20)
    args = (par[:, 0], par[:, 1], par[:, 2], 0.02)
    ref = bayes_fit_gpu(vox, lib, *args, fit_s0=free, quadrature_weights=q)
    side = torch.cuda.Stream()
    M, L = _pending(vox, lib)
    got = bayes_fit_gpu(M, L, *args, fit_s0=free, quadrature_weights=q, stream=side)
    assert set(ref) == set(got)
    for k in ref:
        assert np.array_equal(ref[k], got[k])
