"""The Bayesian fit sums the same entries in the same order with and without the
search index (scratch of madi_bayes_work_bytes or only the column means): equal
outputs bit for bit, also where the bounds could go wrong."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fit(vox, lib, par, logq, free, sigma, small):
    import torch
    from custom_madi_gb300 import _native as N
    n, F = vox.shape
    M, L = torch.from_numpy(vox).cuda(), torch.from_numpy(lib).cuda()
    cols = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (logq, par[:, 0], par[:, 1], par[:, 2])]
    need = int(N.lib().madi_bayes_work_bytes(n, len(lib), F))
    nbytes = int(N.lib().madi_bayes_scratch_bytes(len(lib), F)) if small else need
    buf = torch.empty(nbytes + 256, dtype=torch.uint8, device="cuda")
    out = torch.full((N.MADI_BAYES_N_OUT, n), -7.0, dtype=torch.float64, device="cuda")
    d = N.MadiBayesDesc()
    d.measured, d.lib = N.ptr(M), N.ptr(L)
    d.log_weight, d.kio, d.rho, d.V = (N.ptr(t) for t in cols)
    d.n_vox, d.n_lib, d.n_feat = n, len(lib), F
    d.mode = N.MADI_MATCH_FREE_S0 if free else N.MADI_MATCH_FIXED_S0
    d.sigma_m, d.out = sigma, N.ptr(out)
    base = N.ptr(buf)
    d.scratch, d.scratch_bytes = base + (-base) % 256, nbytes
    N.check(N.lib().madi_bayes(C.byref(d), torch.cuda.current_stream().cuda_stream), "madi_bayes")
    torch.cuda.synchronize()
    return need, out.cpu().numpy()


@pytest.mark.parametrize("free", (False, True))
@pytest.mark.parametrize("n_vox, n_lib, F, kind, sigma", [
    (64, 256, 5, "decays", 0.02), (1_001, 700, 12, "decays", 0.01), (19_456, 300, 17, "masked", 0.05),
    (19_457, 1_025, 20, "decays", 0.02), (700, 513, 24, "nonfinite", 0.02), (700, 513, 32, "constant", 0.02),
    (900, 640, 28, "scales", 0.02),
])
def test_indexed_fit_equals_plain(n_vox, n_lib, F, kind, sigma, free):
    rng = np.random.default_rng(n_vox + F)
    t = np.sort(rng.uniform(0.0, 3.0, F))
    lib = 0.6 * np.exp(-t * rng.uniform(0.1, 3.0, (n_lib, 1))) + 0.4 * np.exp(-t * rng.uniform(0.1, 1.0, (n_lib, 1)))
    vox = lib[rng.integers(0, n_lib, n_vox)] + 0.03 * rng.standard_normal((n_vox, F))
    if free:
        vox *= rng.uniform(200.0, 1500.0, (n_vox, 1))
    if kind == "masked":
        vox[rng.random(n_vox) < 0.6] = 0.0
        lib[::7] = 0.0
    elif kind == "nonfinite":
        vox[5, 0], vox[n_vox // 2, F - 1] = np.nan, np.inf
    elif kind == "constant":
        lib[:] = lib[0]
    elif kind == "scales":
        vox *= 10.0 ** rng.integers(-12, 13, (n_vox, 1))
        lib *= 10.0 ** rng.integers(-4, 5, (n_lib, 1))
    par = np.exp(rng.uniform(np.log([1.0, 4e3, 0.01]), np.log([130.0, 5e7, 200.0]), (n_lib, 3)))
    logq = np.log(rng.uniform(0.2, 1.2, n_lib))
    args = (vox.astype(np.float32), lib.astype(np.float32), par, logq, free, sigma)
    need, a = _fit(*args, small=False)
    assert need > 256
    _, b = _fit(*args, small=True)
    assert np.array_equal(a, b, equal_nan=True)
