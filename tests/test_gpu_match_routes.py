"""The fp32 match picks the same entry on every route: the pruned search and the
split scan (scratch as the library asks) against the plain exhaustive scan (a
scratch that only holds the column means), bit for bit, for ordinary data and for
data on which bounds could go wrong."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _match(vox, lib, free, scratch_bytes=None, flags=4):
    import torch
    from custom_madi_gb300 import _native as N
    M, L = torch.from_numpy(vox).cuda(), torch.from_numpy(lib).cuda()
    n, F = M.shape
    need = int(N.lib().madi_match_scratch_bytes(n, len(lib), F, N.MADI_MATCH_FP32, 32))
    nbytes = need if scratch_bytes is None else scratch_bytes
    buf = torch.full((nbytes + 256,), 0x5A, dtype=torch.uint8, device="cuda")
    out = [torch.full((n,), -7, dtype=torch.int32, device="cuda")] + [torch.zeros(n, device="cuda") for _ in range(2)]
    d = N.MadiMatchDesc()
    d.measured, d.lib, d.n_vox, d.n_lib, d.n_feat = N.ptr(M), N.ptr(L), n, len(lib), F
    d.mode = N.MADI_MATCH_FREE_S0 if free else N.MADI_MATCH_FIXED_S0
    d.precision, d.topk, d.flags = N.MADI_MATCH_FP32, 32, flags
    d.best_idx, d.best_resid, d.best_s0 = (N.ptr(t) for t in out)
    base = N.ptr(buf)
    d.scratch, d.scratch_bytes = base + (-base) % 256, nbytes
    N.check(N.lib().madi_match(C.byref(d), torch.cuda.current_stream().cuda_stream), "madi_match")
    torch.cuda.synchronize()
    if free and not flags:
        assert bool((buf == 0x5A).all())         # the scratch is not this call's to write
    return need, [t.cpu().numpy() for t in out]


def _data(kind, n_vox, n_lib, F, rng):
    t = np.sort(rng.uniform(0.0, 3.0, F))
    rate = rng.uniform(0.1, 3.0, (n_lib, 1))
    lib = 0.6 * np.exp(-t * rate) + 0.4 * np.exp(-t * rng.uniform(0.1, 1.0, (n_lib, 1)))
    vox = lib[rng.integers(0, n_lib, n_vox)] + 0.03 * rng.standard_normal((n_vox, F))
    if kind == "random":                    # nothing to prune
        lib, vox = rng.uniform(0.0, 1.0, (n_lib, F)), rng.uniform(0.0, 1.0, (n_vox, F))
    elif kind == "ties":                    # every entry four times, voxels on entries: lowest index wins
        lib = np.tile(lib[: n_lib // 4], (4, 1))
        lib = lib[rng.permutation(len(lib))]
        vox[::2] = lib[rng.integers(0, len(lib), len(vox[::2]))]
    elif kind == "constant":                # no spread at all, all scores equal
        lib[:] = lib[0]
    elif kind == "masked":                  # background voxels, negative and zero entries
        vox[rng.random(n_vox) < 0.7] = 0.0
        lib[::7] = 0.0
        lib[1::11] *= -1.0
    elif kind == "scales":                  # 1e-18 .. 1e18
        vox *= 10.0 ** rng.integers(-18, 19, (n_vox, 1))
        lib *= 10.0 ** rng.integers(-6, 7, (n_lib, 1))
    elif kind == "nonfinite":
        vox[5, 0], vox[n_vox // 2, F - 1], vox[n_vox - 1, 0] = np.nan, np.inf, -np.inf
        lib[3, 0], lib[n_lib // 2, F - 1] = np.nan, np.inf
    elif kind == "nonfinite voxels":
        vox[5, 0], vox[n_vox // 2, F - 1], vox[n_vox - 1, 0] = np.nan, np.inf, -np.inf
    return vox.astype(np.float32), lib.astype(np.float32)


KINDS = ("decays", "random", "ties", "constant", "masked", "scales", "nonfinite", "nonfinite voxels")


@pytest.mark.parametrize("free", (False, True))
@pytest.mark.parametrize("kind", KINDS)
def test_pruned_search_equals_scan(kind, free):
    for n_vox, n_lib, F in ((50_001, 4_099, 20), (130_000, 1_025, 31), (300_001, 1_025, 14)):   # 4, 2, 1 warps a group
        vox, lib = _data(kind, n_vox, n_lib, F, np.random.default_rng(n_lib + F))
        need, a = _match(vox, lib, free)
        assert need > 256 + 8 * n_vox           # the index: this size is pruned
        _, b = _match(vox, lib, free, scratch_bytes=256)
        for x, y in zip(a, b):
            assert np.array_equal(x, y, equal_nan=True)


@pytest.mark.parametrize("free", (False, True))
@pytest.mark.parametrize("n_vox, n_lib, F, kind", [
    (1, 8, 4, "decays"), (1, 129, 2, "decays"), (127, 128, 5, "ties"), (129, 5_000, 10, "masked"),
    (3_001, 5_000, 12, "ties"), (2_000, 257, 32, "nonfinite"), (200_000, 300, 8, "decays"), (400_001, 257, 28, "decays"),
])
def test_split_scan_equals_scan(n_vox, n_lib, F, kind, free):
    vox, lib = _data(kind, n_vox, n_lib, F, np.random.default_rng(n_vox + F))
    _, a = _match(vox, lib, free)
    _, b = _match(vox, lib, free, scratch_bytes=256)
    for x, y in zip(a, b):
        assert np.array_equal(x, y, equal_nan=True)


@pytest.mark.parametrize("n_vox, n_lib, F", [(50_001, 4_099, 20), (3_001, 5_000, 12)])
def test_free_s0_leaves_the_scratch_alone_without_the_flag(n_vox, n_lib, F):
    vox, lib = _data("decays", n_vox, n_lib, F, np.random.default_rng(1))
    _, a = _match(vox, lib, True)
    _, b = _match(vox, lib, True, flags=0)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
