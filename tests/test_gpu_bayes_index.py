"""The Bayesian fit on both sides of the line from which it takes its search index, and
the index where bounds could go wrong: the sums of the fit without it, bit for bit."""

import numpy as np
import pytest

from test_gpu_bayes_routes import _fit

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("free", (False, True))
@pytest.mark.parametrize("n_vox, n_lib, F, kind, sigma", [
    (63, 1_000, 5, "decays", 0.02), (64, 1_000, 5, "decays", 0.02), (65, 999, 5, "decays", 0.02), (1_001, 1_000, 12, "decays", 0.01),
    (19_455, 1_000, 17, "masked", 0.05), (19_456, 400, 17, "masked", 0.05), (19_456, 399, 17, "masked", 0.05),
    (700, 1_025, 24, "nonfinite", 0.02), (700, 1_025, 32, "constant", 0.02), (900, 1_280, 28, "scales", 0.02),
    (20_000, 1_500, 8, "scales", 0.02), (20_000, 513, 24, "nonfinite", 0.02),
])
def test_both_sides_of_the_line(n_vox, n_lib, F, kind, sigma, free):
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
        lib[11, 0], lib[n_lib // 2, F - 1] = np.nan, np.inf
    elif kind == "constant":
        lib[:] = lib[0]
    elif kind == "scales":
        vox *= 10.0 ** rng.integers(-12, 13, (n_vox, 1))
        lib *= 10.0 ** rng.integers(-4, 5, (n_lib, 1))
    par = np.exp(rng.uniform(np.log([1.0, 4e3, 0.01]), np.log([130.0, 5e7, 200.0]), (n_lib, 3)))
    logq = np.log(rng.uniform(0.2, 1.2, n_lib))
    args = (vox.astype(np.float32), lib.astype(np.float32), par, logq, free, sigma)
    _, a = _fit(*args, small=False)
    _, b = _fit(*args, small=True)
    assert np.array_equal(a, b, equal_nan=True)


@pytest.mark.parametrize("n_vox, n_lib, index", [(500, 256, False), (19_455, 999, False), (64, 1_000, True), (19_456, 399, False),
                                                 (19_456, 400, True)])
def test_the_index_is_taken_only_where_it_pays(n_vox, n_lib, index):
    """Seen by whether the scratch behind the column means is written."""
    import ctypes as C
    import torch
    from custom_madi_gb300 import _native as N
    M, L = torch.rand((n_vox, 20), device="cuda"), torch.rand((n_lib, 20), device="cuda")
    par = torch.rand((4, n_lib), dtype=torch.float64, device="cuda")
    out = torch.empty((N.MADI_BAYES_N_OUT, n_vox), dtype=torch.float64, device="cuda")
    need = int(N.lib().madi_bayes_work_bytes(n_vox, n_lib, 20))
    buf = torch.full((need + 256,), 0x5A, dtype=torch.uint8, device="cuda")
    d = N.MadiBayesDesc()
    d.measured, d.lib = N.ptr(M), N.ptr(L)
    d.log_weight, d.kio, d.rho, d.V = (N.ptr(par[k]) for k in range(4))
    d.n_vox, d.n_lib, d.n_feat, d.mode, d.sigma_m, d.out = n_vox, n_lib, 20, N.MADI_MATCH_FIXED_S0, 0.02, N.ptr(out)
    pad = (-N.ptr(buf)) % 256
    d.scratch, d.scratch_bytes = N.ptr(buf) + pad, need
    N.check(N.lib().madi_bayes(C.byref(d), torch.cuda.current_stream().cuda_stream), "madi_bayes")
    torch.cuda.synchronize()
    assert bool((buf[pad + 256:] != 0x5A).any()) == index
