"""madi_classify (through the C ABI) against the reference's labels: bit-exact."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _classify(ens, pts, method, f32):
    import torch
    from custom_madi_gb300 import _native as N
    dev = ens.device()
    p = torch.from_numpy(np.ascontiguousarray(pts, np.float32 if f32 else np.float64)).cuda()
    n = len(pts)
    cell = torch.empty(n, dtype=torch.int32, device="cuda")
    inside = torch.empty(n, dtype=torch.uint8, device="cuda")
    path = torch.empty(n, dtype=torch.uint8, device="cuda")
    st = N.lib().madi_classify(C.byref(dev.struct), N.ptr(p), 1 if f32 else 0, n, method, N.ptr(cell),
                               N.ptr(inside), N.ptr(path), torch.cuda.current_stream().cuda_stream)
    N.check(st, "madi_classify")
    torch.cuda.synchronize()
    return cell.cpu().numpy(), inside.cpu().numpy().astype(bool), path.cpu().numpy()


def _si_ensemble(d):
    from custom_madi_gb300.ensemble import ensemble_from_arrays
    return ensemble_from_arrays(d["seeds"], d["annulus"], float(d["L"]), source_lo=float(d["source_lo"]),
                                source_hi=float(d["source_hi"]), rho_per_uL=float(d["rho"]))


def test_kd_fp64_bit_exact_vs_reference(golden):
    d = golden("classify_si.npz")
    ens = _si_ensemble(d)
    assert np.array_equal(ens.kd_node_seed, d["kd_node_seed"])
    c, i, path = _classify(ens, d["points"], 0, False)
    assert np.array_equal(c, d["cell"]) and np.array_equal(i, d["inside"])
    assert np.all(path == 2)


@pytest.mark.parametrize("pts,cell,inside", [("points32", "cell32", "inside32"), ("near32", "cell_near32", "inside_near32")])
def test_grid_fp32_bit_exact_vs_reference(golden, pts, cell, inside):
    d = golden("classify_si.npz")
    ens = _si_ensemble(d)
    c, i, path = _classify(ens, d[pts], 1, True)
    assert np.array_equal(c, d[cell]) and np.array_equal(i, d[inside])
    assert np.mean(path == 1) < 0.05       # fp64 fallbacks are rare
    assert np.all(path != 255)
    c64, i64, _ = _classify(ens, d[pts], 1, False)
    assert np.array_equal(c64, d[cell]) and np.array_equal(i64, d[inside])


def test_grid_periodic_bit_exact_vs_27_image_reference(golden):
    from custom_madi_gb300.ensemble import ensemble_from_arrays
    d = golden("classify_periodic.npz")
    ens = ensemble_from_arrays(d["base_seeds"], d["annulus"], float(d["L"]), source_lo=0.0, source_hi=float(d["L"]),
                               rho_per_uL=float(d["rho"]), boundary_mode="periodic")
    for method, f32 in ((1, True), (0, False), (1, False)):
        c, i, _ = _classify(ens, d["points"], method, f32)
        assert np.array_equal(i, d["inside"]), (method, f32)
        assert np.array_equal(c, d["cell"]), (method, f32)


def test_classify_random_stream_vs_oracle_large():
    """2e5 random fp32 points of a fresh periodic ensemble: device == oracle brute force."""
    from custom_madi_gb300.config import SimConfig
    from custom_madi_gb300.ensemble import create_ensemble
    from oracle import oracle as O
    cfg = SimConfig(boundary_mode="periodic", n_cells=100, ts=0.01, T_max_ms=46.0, small_deltas=[6.0],
                    big_deltas=[15.0, 25.0, 30.0, 40.0], geometry_validation_points=20000, geometry_vi_tolerance=0.05)
    ens = create_ensemble(3.0e5, 0.9 * 1e6 / 3.0e5, cfg, seed=11)
    pts = np.random.default_rng(5).uniform(0, ens.L, size=(200_000, 3)).astype(np.float32).astype(np.float64)
    c, i, path = _classify(ens, pts, 1, True)
    oc, oi = O.classify_kd(O.geom_arrays(ens), pts)
    assert np.array_equal(i, oi) and np.array_equal(c, oc)
    assert np.mean(path == 1) < 0.01


@pytest.mark.parametrize("mode, n_cells, rho, V", [("periodic", 2, 2.0e5, 4.0), ("periodic", 300, 5.0e7, 0.017),
                                                   ("si_fatal_escape", 0, 1.0e5, 7.0)])
def test_fp64_points_in_fp32_band(mode, n_cells, rho, V):
    """fp64 points decided in fp32 where the band allows: the labels of the KD rule,
    also on and within rounding of shifted facets, seeds and box faces."""
    from custom_madi_gb300.config import SimConfig
    from custom_madi_gb300.ensemble import create_ensemble
    over = dict(boundary_mode="periodic", n_cells=n_cells) if mode == "periodic" else {}
    cfg = SimConfig(n_ensembles=1, ts=0.01, T_max_ms=4.0, small_deltas=[1.0], big_deltas=[2.0], b_values=[0.0, 1000.0], **over)
    ens = create_ensemble(rho, V, cfg, seed=9, verify_vi=False, measure_vi=False)
    rng = np.random.default_rng(4)
    p = rng.uniform(0.0, ens.L, size=(20_000, 3))
    cs = ens.classifier_seeds if ens.classifier_seeds is not None else ens.seeds
    an = ens.classifier_annulus if ens.classifier_annulus is not None else ens.annulus
    i, j = rng.integers(0, len(cs), 5_000), rng.integers(0, len(cs), 5_000)
    u = cs[j] - cs[i]
    d = np.maximum(np.linalg.norm(u, axis=1, keepdims=True), 1e-12)
    on = cs[i] + u * (0.5 - an[i][:, None] / d)                       # on the shifted facet of (i, j)
    near = on + 10.0 ** rng.uniform(-13, -4, (len(on), 1)) * rng.standard_normal(on.shape)
    q = np.concatenate([p, on, near, cs[i], np.where(rng.random(p.shape) < 0.3, 0.0, p)])
    q = q[np.all((q >= 0.0) & (q < ens.L), axis=1)]
    a, b = ens.classify(q, method="grid"), ens.classify(q, method="kd")
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
