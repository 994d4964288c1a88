// Pruned library search: an exact argmin that skips library tiles which cannot
// hold the winner.
//
// Rows x (fixed S0: centred on the library mean; free S0: unit rows, centred)
// are embedded as Phi(x) = (v_1.x, .., v_5.x, |x - sum (v_k.x) v_k|) with v_k
// orthonormal, leading directions of a sample of the library.  Phi is
// 1-Lipschitz, so the distance from Phi(voxel) to the box of a tile's Phi
// values bounds the distance from the voxel to each of the tile's entries from
// below, whatever the directions are: they decide how many tiles are skipped,
// never the result.  Library entries are put in slabs along v_1, by v_2 inside a
// slab, and cut into tiles of TILE; voxels are ordered by (v_1, v_2, v_3) buckets
// so that the voxels of a warp need the same tiles.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstdint>
#include "madi_device.cuh"
#include "madi_host.h"

namespace madi {
namespace prune {

constexpr int TILE = 32;                        // library entries per tile
constexpr int KDIR = 5;                         // directions of the embedding
constexpr int FMAX = 32;
constexpr int SAMPLE = 512;                     // rows sampled for the directions and ranges
constexpr int LIB_FINE = 512;                   // v_2 buckets of a slab
constexpr int MAX_SLABS = 64;
constexpr int MAX_LIB = 1 << 30;                // entries: rounded up to tiles and blocks they stay in 32 bits
constexpr int LIB_BINS = MAX_SLABS * LIB_FINE;
constexpr int VOX_BINS = 64 * 32 * 16;          // (v_1, v_2, v_3) buckets

struct Phi { float p[KDIR], q; };

// Device arrays, all inside the caller's scratch.
struct Index {
    const float* mu;            // [32] subtracted from the row (fixed S0), or null
    float* basis;               // [KDIR][32] directions, [32] centre of unit rows (free S0), ranges
    float* lmax;                // largest |row|^2; free S0: then the largest 1 / max(|row|^2, 1e-30)
    int* status;                // 0, or a bounded wait of the search ran out (match.cu)
    uint32_t* bins;             // [LIB_BINS + VOX_BINS]
    uint32_t* lbin;             // [n_lib]
    uint32_t* vbin;             // [n_vox]
    int32_t* lperm;             // [n_tiles * TILE] library index, ascending inside a tile, -1 pads
    int32_t* vperm;             // [n_vox]
    float* phi;                 // [n_lib][8]
    float* rows;                // [n_tiles * TILE][row stride]
    float* box;                 // [n_tiles][16]: low 6, high 6 of the tile's Phi
    int64_t n_vox;
    int n_lib, F, n_tiles, slabs, stride;
    int free_s0;
    int test_stall;             // tests only: one wait that nothing completes
};

constexpr int B_CENTRE = KDIR * FMAX, B_RANGE = B_CENTRE + FMAX, B_FLOATS = B_RANGE + 16;

// row padded to a multiple of 4 (at least 8), then |row|^2 and the library index
inline int row_stride(int F) { return (F <= 8 ? 8 : (F + 3) / 4 * 4) + 4; }

// Layout of the index at `base` (256-byte aligned); with base = nullptr only the size is meant.
inline int64_t layout(Index& ix, unsigned char* base, int64_t n_vox, int32_t n_lib, int32_t F) {
    int64_t at = 0;
    auto take = [&](int64_t bytes) {
        unsigned char* p = base + at;
        at += (bytes + 255) / 256 * 256;
        return p;
    };
    ix.n_vox = n_vox;
    ix.n_lib = n_lib;
    ix.F = F;
    ix.n_tiles = (n_lib + TILE - 1) / TILE;
    ix.slabs = (int)std::min<double>(MAX_SLABS, std::max(4.0, 2.5 * std::sqrt((double)ix.n_tiles)));
    ix.mu = nullptr;
    ix.free_s0 = 0;
    ix.test_stall = 0;
    ix.stride = row_stride(F);
    ix.basis = reinterpret_cast<float*>(take(B_FLOATS * 4));
    ix.bins = reinterpret_cast<uint32_t*>(take((LIB_BINS + VOX_BINS) * 4 + 256));
    ix.lmax = reinterpret_cast<float*>(ix.bins + LIB_BINS + VOX_BINS);      // zeroed with the bins
    ix.status = reinterpret_cast<int*>(ix.lmax + 2);                        // so is the status
    ix.lbin = reinterpret_cast<uint32_t*>(take(4ll * n_lib));
    ix.vbin = reinterpret_cast<uint32_t*>(take(4ll * n_vox));
    ix.lperm = reinterpret_cast<int32_t*>(take(4ll * ix.n_tiles * TILE));
    ix.vperm = reinterpret_cast<int32_t*>(take(4ll * n_vox));
    ix.phi = reinterpret_cast<float*>(take(32ll * n_lib));
    ix.rows = reinterpret_cast<float*>(take(4ll * ix.n_tiles * TILE * ix.stride));
    ix.box = reinterpret_cast<float*>(take(64ll * ix.n_tiles));
    return at;
}

// Enqueues the kernels that fill the index: directions, embedding of the library,
// voxel order and, with `tiles`, the library order, rows and boxes.
madi_status build(const Index& ix, const float* meas, const float* lib, bool tiles, cudaStream_t s);

// Embedding of a row x[0..F) (already centred / scaled); v = basis in shared memory.
template <int N>
MADI_DEV Phi embed(const float (&x)[N], const float* v) {
    Phi e;
#pragma unroll
    for (int k = 0; k < KDIR; ++k) {
        float a = 0.f;
#pragma unroll
        for (int f = 0; f < N; ++f) a = fmaf(x[f], v[k * FMAX + f], a);
        e.p[k] = a;
    }
    float q = 0.f;
#pragma unroll
    for (int f = 0; f < N; ++f) {
        float r = x[f];
#pragma unroll
        for (int k = 0; k < KDIR; ++k) r = fmaf(-e.p[k], v[k * FMAX + f], r);
        q = fmaf(r, r, q);
    }
    e.q = sqrtf(q);
    return e;
}

}  // namespace prune
}  // namespace madi
