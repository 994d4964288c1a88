// Library match (MAP nearest library entry per voxel), replacing
// _map_kernel_fixed / _map_kernel_free_s0 (madi/fitters_gpu.py:96-154).
//
// FP32 path, fp32 scores on the CUDA cores.  Fixed S0 scores the centred pair
// (m - mu, L_j - mu), mu the library column mean: the uncentred expanded form
// |L_j|^2 - 2 m.L_j rounds at ~|L|^2 2^-24, coarser than the gap between
// near-tied entries of a dense library, while the centred form rounds at
// ~|L - mu|^2 2^-24.  The choice is the lowest score, the lowest index among
// equal ones, whichever kernel finds it:
//   match_pruned_kernel  large fits: library tiles that cannot hold the winner
//                        are skipped (prune.cuh);
//   match_scan_kernel    every pair; small fits split the library over CTAs.
#include <algorithm>
#include <cstdint>
#include "madi_device.cuh"
#include "madi_host.h"
#include "prune.cuh"

namespace madi {

constexpr int MATCH_THREADS = 128;
constexpr int MATCH_CHUNK = 128;
constexpr float NO_SCORE = 3.0e38f;

// (score, index) as one word that orders like the pair; -0 and 0 are equal scores.
MADI_DEV unsigned long long match_key(float score, int j) {
    const uint32_t o = (uint32_t)f2o(score + 0.0f) ^ 0x80000000u;
    return ((unsigned long long)o << 32) | (uint32_t)j;
}

// Residual of the chosen entry from the direct difference of the raw data.
template <int N, int MODE>
MADI_DEV void match_write(const float* __restrict__ meas, const float* __restrict__ lib, int64_t v, int bj, int n_feat,
                          int32_t* best_idx, float* best_resid, float* best_s0) {
    const float* M = meas + v * n_feat;
    const float* L = lib + (int64_t)bj * n_feat;
    float dot = 0.f, rr = 0.f;
#pragma unroll
    for (int f = 0; f < N; ++f) {
        if (f < n_feat) { dot = fmaf(M[f], L[f], dot); rr = fmaf(L[f], L[f], rr); }
    }
    float s0 = 1.f;
    if (MODE == MADI_MATCH_FREE_S0) s0 = dot / fmaxf(rr, 1e-30f);
    float res = 0.f;
#pragma unroll
    for (int f = 0; f < N; ++f) {
        if (f < n_feat) {
            const float r = M[f] - s0 * L[f];
            res = fmaf(r, r, res);
        }
    }
    if (MODE == MADI_MATCH_FREE_S0 && !(dot > 0.f)) res = 3.0e38f;
    best_idx[v] = bj;
    best_resid[v] = res;
    if (MODE == MADI_MATCH_FREE_S0 && best_s0) best_s0[v] = s0;
}

// Fixed S0 score_j = |L_j - mu|^2 - 2 (m - mu).(L_j - mu) = |m - L_j|^2 - |m - mu|^2;
// free S0 score_j = -(m.r)^2 / |r|^2 when m.r > 0.  The free score's division is
// only made for pairs that may reach the best so far: dot^2 >= bar |r|^2, bar
// 4e-7 below the best (the rounding on both sides is below 2e-7), 0 where the
// best is subnormal or there is none.  An entry whose |r|^2 overflows (bar |r|^2
// infinite, or NaN with the bar 0) is left to the score itself.
MADI_DEV float free_bar(float best) { return best < -1e-36f ? -best * (1.f - 4e-7f) : 0.f; }
MADI_DEV bool free_may_win(float dot, float sn, float bar) {
    return dot > 0.f && !(fmaxf(dot * dot, 1e-36f) < bar * sn);
}

template <int MODE>
MADI_DEV void match_pair(float dot, float sn, int j, float& best, int& bj, float& bar) {
    if (MODE == MADI_MATCH_FIXED_S0) {
        const float score = fmaf(-2.f, dot, sn);
        if (score < best) { best = score; bj = j; }
    } else if (free_may_win(dot, sn, bar)) {
        const float score = -(dot * dot) / sn;
        if (score < best) { best = score; bj = j; bar = free_bar(best); }
    }
}

// Every pair: the library (or the part blockIdx.y of it) streams through shared
// memory, V voxels per thread so that one 16-byte shared load feeds 4 V fused
// multiply-adds (with one voxel a thread the shared-memory pipe, not the FMA
// pipe, was the limit).  keys != null: the part's winners meet in a 64-bit
// minimum per voxel and match_finish_kernel writes the results.
template <int N, int MODE, int V>
__global__ void __launch_bounds__(MATCH_THREADS) match_scan_kernel(const float* __restrict__ meas,
                                                                   const float* __restrict__ lib,
                                                                   const float* __restrict__ mu, int64_t n_vox,
                                                                   int n_lib, int n_feat, int part,
                                                                   unsigned long long* keys, int32_t* best_idx,
                                                                   float* best_resid, float* best_s0) {
    __shared__ float4 sl[MATCH_CHUNK][N / 4];
    __shared__ float sn[MATCH_CHUNK];
    __shared__ float smu[N];
    const int64_t v0 = (int64_t)blockIdx.x * (MATCH_THREADS * V) + threadIdx.x;
    if (threadIdx.x < N)
        smu[threadIdx.x] = (MODE == MADI_MATCH_FIXED_S0 && (int)threadIdx.x < n_feat) ? mu[threadIdx.x] : 0.f;
    __syncthreads();
    float m[V][N];
    float best[V], bar[V];
    int bj[V];
#pragma unroll
    for (int i = 0; i < V; ++i) {
        const int64_t v = v0 + i * MATCH_THREADS;
#pragma unroll
        for (int f = 0; f < N; ++f) m[i][f] = (v < n_vox && f < n_feat) ? meas[v * n_feat + f] - smu[f] : 0.f;
        best[i] = NO_SCORE;
        bar[i] = 0.f;
        bj[i] = 0;
    }
    const int j0 = blockIdx.y * part, j1 = n_lib - j0 > part ? j0 + part : n_lib;
    float* flat = reinterpret_cast<float*>(sl);
    for (int t = threadIdx.x; t < MATCH_CHUNK * (N - n_feat); t += MATCH_THREADS) {      // never written again
        const int e = t / (N - n_feat), f = n_feat + t - e * (N - n_feat);
        flat[e * N + f] = 0.f;
    }
    // a thread's place in the rows moves by (de, df) from one of its loads to the next
    const int e0 = threadIdx.x / n_feat, f0 = threadIdx.x - e0 * n_feat;
    const int de = MATCH_THREADS / n_feat, df = MATCH_THREADS - de * n_feat;
    for (unsigned base = j0; base < (unsigned)j1; base += MATCH_CHUNK) {
        const int cnt = min(MATCH_CHUNK, j1 - (int)base);
        __syncthreads();
        const float* src = lib + (int64_t)base * n_feat;
        int e = e0, f = f0;
        constexpr int AHEAD = 4;                                // loads in flight (2: +5 %, 8: +12 % at two voxels a thread)
        for (int t0 = threadIdx.x; t0 < cnt * n_feat; t0 += AHEAD * MATCH_THREADS) {
            float x[AHEAD];
#pragma unroll
            for (int i = 0; i < AHEAD; ++i) {
                const int t = t0 + i * MATCH_THREADS;
                x[i] = t < cnt * n_feat ? src[t] : 0.f;
            }
#pragma unroll
            for (int i = 0; i < AHEAD; ++i) {
                if (t0 + i * MATCH_THREADS < cnt * n_feat) flat[e * N + f] = x[i] - smu[f];
                e += de;
                f += df;
                if (f >= n_feat) { f -= n_feat; ++e; }
            }
        }
        __syncthreads();
        if ((int)threadIdx.x < cnt) {
            float s = 0.f;
#pragma unroll
            for (int f = 0; f < N / 4; ++f) {
                const float4 l = sl[threadIdx.x][f];
                s = fmaf(l.x, l.x, s); s = fmaf(l.y, l.y, s); s = fmaf(l.z, l.z, s); s = fmaf(l.w, l.w, s);
            }
            sn[threadIdx.x] = MODE == MADI_MATCH_FREE_S0 ? fmaxf(s, 1e-30f) : s;
        }
        __syncthreads();
        // entries ahead: with few warps an SM their chains are the time (5,000 entries x 10,
        // one voxel a thread, two / four at a time: 342 / 206 us)
#pragma unroll (V == 1 && N > 8 ? 4 : 2)
        for (int e = 0; e < cnt; ++e) {
            float dot[V];
#pragma unroll
            for (int i = 0; i < V; ++i) dot[i] = 0.f;
#pragma unroll
            for (int f = 0; f < N / 4; ++f) {
                const float4 l = sl[e][f];
#pragma unroll
                for (int i = 0; i < V; ++i) {
                    dot[i] = fmaf(m[i][4 * f], l.x, dot[i]);
                    dot[i] = fmaf(m[i][4 * f + 1], l.y, dot[i]);
                    dot[i] = fmaf(m[i][4 * f + 2], l.z, dot[i]);
                    dot[i] = fmaf(m[i][4 * f + 3], l.w, dot[i]);
                }
            }
#pragma unroll
            for (int i = 0; i < V; ++i) match_pair<MODE>(dot[i], sn[e], (int)base + e, best[i], bj[i], bar[i]);
        }
    }
#pragma unroll
    for (int i = 0; i < V; ++i) {
        const int64_t v = v0 + i * MATCH_THREADS;
        if (v >= n_vox) continue;
        if (keys) atomicMin(&keys[v], match_key(best[i], bj[i]));
        else match_write<N, MODE>(meas, lib, v, bj[i], n_feat, best_idx, best_resid, best_s0);
    }
}

template <int N, int MODE>
__global__ void __launch_bounds__(256) match_finish_kernel(const float* __restrict__ meas, const float* __restrict__ lib,
                                                           const unsigned long long* __restrict__ keys, int64_t n_vox,
                                                           int n_feat, int32_t* best_idx, float* best_resid,
                                                           float* best_s0) {
    const int64_t v = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (v < n_vox) match_write<N, MODE>(meas, lib, v, (int)(uint32_t)keys[v], n_feat, best_idx, best_resid, best_s0);
}

// ---------------------------------------------------------------------------
// Pruned search.  A group of 64 voxels that are neighbours in the index's order
// (two per lane) has the tile nearest to it scanned, then every tile that some
// voxel still needs: first by the box of the group's voxels (32 tiles at a time,
// one per lane), then voxel by voxel.  A tile's rows (6 KB at 20 features) come
// to shared memory by one bulk copy while the tile before is scanned: read in
// place, each entry waited for its 6 broadcast loads.  WARPS warps share a
// group's tiles and merge their winners, so that small fits fill the chip.
//
// Why nothing is missed: with d the box distance in the embedding, every entry
// of the tile has |m - L|^2 >= d^2 (1-Lipschitz), so its exact score is at least
// d^2 - |m|^2 (fixed S0), and |cos| <= 1 - d^2 / 2 between unit rows (free S0).
// The fp32 score is off by at most (F + 2) 2^-24 (|m|^2 + 2 |L|^2) (two dot
// products), the fp32 embedding by (F + 8) 2^-23 (|m| + |L|) per coordinate, and
// the directions are orthonormal to 1e-5: 0.998 d^2 and the margin E = (F + 8)
// 2^-21 (|m|^2 + max |L|^2) cover them together ((a + b)^2 <= 1.001 a^2 + 1001
// b^2).  A tile is skipped only if the bound lies strictly above the best score,
// so ties keep the lowest index.  Where fp32 scores can overflow or the terms of
// the bounds become subnormal (rounded by an absolute amount, which no relative
// margin covers), the bound says nothing: those voxels (and ones that are not
// finite) skip nothing.
// ---------------------------------------------------------------------------
struct PrunedVoxel {
    float m2, e, limit, best;
    int bj;
    bool bounded;
};

template <int MODE>
MADI_DEV void set_limit(PrunedVoxel& v) {
    if (MODE == MADI_MATCH_FIXED_S0) {
        v.limit = v.best + v.m2 + v.e;
    } else {
        const float s = v.best < 0.f ? fmaxf(-v.best / v.m2 - v.e, 0.f) : 0.f;     // cos^2 to beat
        v.limit = 2.f * (1.f - sqrtf(s)) + 4e-6f;
    }
    if (!v.bounded || !(v.limit < NO_SCORE)) v.limit = __int_as_float(0x7f800000);
}

MADI_DEV float warp_minf32(float v) { float r; asm("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v)); return r; }
MADI_DEV float warp_maxf32(float v) { float r; asm("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v)); return r; }

// Squared distance between the boxes [lo, hi] and the tile's.
MADI_DEV float box_distance2(const float4* __restrict__ b, const float (&lo)[6], const float (&hi)[6]) {
    const float4 l0 = b[0], l1 = b[1], h0 = b[2], h1 = b[3];
    const float tl[6] = {l0.x, l0.y, l0.z, l0.w, l1.x, l1.y}, th[6] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y};
    float d2 = 0.f;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        const float d = fmaxf(fmaxf(tl[k] - hi[k], lo[k] - th[k]), 0.f);
        d2 = fmaf(d, d, d2);
    }
    return d2;
}

// Scores a tile for the two voxels of every lane.  Rows come in pairs of entries,
// feature by feature, so one packed instruction advances both entries' dot
// products (m holds each feature twice).
template <int N, int MODE>
MADI_DEV void scan_tile(const ulonglong2* rows, const uint64_t (&ma)[N], const uint64_t (&mb)[N], PrunedVoxel& a,
                        PrunedVoxel& b) {
    // winners of the tile alone (its entries are in index order), then against the
    // best so far; the free score's bar starts from the best so far
    float ta = NO_SCORE, tb = NO_SCORE;
    float bara = MODE == MADI_MATCH_FIXED_S0 ? 0.f : free_bar(a.best), barb = MODE == MADI_MATCH_FIXED_S0 ? 0.f : free_bar(b.best);
    int ja = -1, jb = -1;
#pragma unroll 2
    for (int e = 0; e < prune::TILE / 2; ++e) {
        const ulonglong2* r = rows + e * (N / 2 + 2);
        uint64_t da = 0, db = 0;
#pragma unroll
        for (int f = 0; f < N / 2; ++f) {
            const ulonglong2 l = r[f];
            da = fma2(ma[2 * f], l.x, da); da = fma2(ma[2 * f + 1], l.y, da);
            db = fma2(mb[2 * f], l.x, db); db = fma2(mb[2 * f + 1], l.y, db);
        }
        const ulonglong2 x = r[N / 2];
        const float2 sn = split2(x.x), id = split2(x.y), ea = split2(da), eb = split2(db);
        match_pair<MODE>(ea.x, sn.x, __float_as_int(id.x), ta, ja, bara);
        match_pair<MODE>(eb.x, sn.x, __float_as_int(id.x), tb, jb, barb);
        match_pair<MODE>(ea.y, sn.y, __float_as_int(id.y), ta, ja, bara);
        match_pair<MODE>(eb.y, sn.y, __float_as_int(id.y), tb, jb, barb);
    }
    if (ja >= 0 && (ta < a.best || (ta == a.best && ja < a.bj))) { a.best = ta; a.bj = ja; }
    if (jb >= 0 && (tb < b.best || (tb == b.best && jb < b.bj))) { b.best = tb; b.bj = jb; }
    set_limit<MODE>(a);
    set_limit<MODE>(b);
}

// Bulk copy of one tile's rows into shared memory, completing on `bar`.
MADI_DEV void tile_fetch(float4* dst, const float4* src, uint32_t bytes, uint64_t* bar) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst), b = (uint32_t)__cvta_generic_to_shared(bar);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(b), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 :: "r"(d), "l"(src), "r"(bytes), "r"(b) : "memory");
}

// Waits for phase `parity` of a tile copy, ~1 s at most (20 us suspends); false in
// every lane if it ran out for one.
constexpr int WAIT_POLLS = 50000;
constexpr int STALL_POLLS = 64;                 // the test-only stalled wait (MADI_MATCH_FLAG_TEST_STALL)
MADI_DEV bool tile_wait(uint64_t* bar, uint32_t parity, int polls = WAIT_POLLS) {
    const uint32_t b = (uint32_t)__cvta_generic_to_shared(bar);
    uint32_t done = 0;
    for (int i = 0; i < polls && !done; ++i)
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}"
                     : "=r"(done) : "r"(b), "r"(parity), "r"(20000u) : "memory");
    return __all_sync(MADI_FULL, done);
}

template <int N, int MODE, int WARPS>
__global__ void __launch_bounds__(MATCH_THREADS, N <= 12 ? 4 : N <= 24 ? 3 : 2) match_pruned_kernel(const float* __restrict__ meas,
                                                                        const float* __restrict__ lib,
                                                                        const prune::Index ix, int32_t* best_idx,
                                                                        float* best_resid, float* best_s0) {
    constexpr int NW = MATCH_THREADS / 32, GROUPS = NW / WARPS;
    constexpr int TILE4 = prune::TILE * (N / 4 + 1);                           // float4 of a tile's rows
    extern __shared__ __align__(128) float4 stage[];                           // [warp][2][TILE4]
    __shared__ float sv[prune::B_FLOATS], smu[N];
    __shared__ uint64_t bars[NW][2], never;                                    // never: no thread arrives (tests)
    __shared__ unsigned long long merged[WARPS > 1 ? GROUPS : 1][64];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < prune::B_FLOATS; i += MATCH_THREADS) sv[i] = ix.basis[i];
    if (threadIdx.x < N)
        smu[threadIdx.x] = (MODE == MADI_MATCH_FIXED_S0 && (int)threadIdx.x < ix.F) ? ix.mu[threadIdx.x] : 0.f;
    if (WARPS > 1)
        for (int i = threadIdx.x; i < GROUPS * 64; i += MATCH_THREADS) merged[i >> 6][i & 63] = ~0ull;
    if (lane < 2) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"((uint32_t)__cvta_generic_to_shared(&bars[warp][lane])) : "memory");
    if (threadIdx.x == 0) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"((uint32_t)__cvta_generic_to_shared(&never)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    __syncthreads();
    const int64_t p0 = ((int64_t)blockIdx.x * GROUPS + warp / WARPS) * 64;
    const int part = warp % WARPS;
    const bool live = p0 < ix.n_vox;                                           // a whole group
    if (WARPS == 1 && !live) return;
    const float slack = (float)(ix.F + 8) * 4.76837158203125e-07f;             // (F + 8) 2^-21
    const float lmax = ix.lmax[0], inv_lmin = ix.lmax[1];
    int64_t vox[2];
    PrunedVoxel pv[2];
    if (live) {
        uint64_t mm[2][N];
        float phi[2][6];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            float m[N];
            vox[i] = ix.vperm[min(p0 + 32 * i + lane, ix.n_vox - 1)];
            PrunedVoxel& v = pv[i];
            v.m2 = 0.f;
#pragma unroll
            for (int f = 0; f < N; ++f) {
                m[f] = f < ix.F ? meas[vox[i] * ix.F + f] - smu[f] : 0.f;
                v.m2 = fmaf(m[f], m[f], v.m2);
            }
            prune::Phi e;
            if (MODE == MADI_MATCH_FIXED_S0) {
                e = prune::embed(m, sv);
                v.e = slack * (v.m2 + lmax);
                v.bounded = v.m2 + lmax < 1e36f && v.m2 + lmax > 1e-30f;
            } else {
                float u[N];
                const float sc = v.m2 > 0.f ? rsqrtf(v.m2) : 0.f;
#pragma unroll
                for (int f = 0; f < N; ++f) u[f] = f < ix.F ? fmaf(m[f], sc, -sv[prune::B_CENTRE + f]) : 0.f;
                e = prune::embed(u, sv);
                v.e = slack;
                v.bounded = v.m2 < 1e36f && v.m2 * lmax < 1e36f && v.m2 > 1e-32f * inv_lmin && inv_lmin < 1e25f;
            }
#pragma unroll
            for (int k = 0; k < prune::KDIR; ++k) phi[i][k] = e.p[k];
            phi[i][5] = e.q;
#pragma unroll
            for (int f = 0; f < N; ++f) mm[i][f] = pair2(m[f], m[f]);
            v.best = NO_SCORE;
            v.bj = 0;
            set_limit<MODE>(v);
        }
        const float4* boxes = reinterpret_cast<const float4*>(ix.box);
        const float4* rows = reinterpret_cast<const float4*>(ix.rows);
        float4* buf = stage + warp * 2 * TILE4;
        uint32_t fetched = 0, scanned = 0;                                     // tiles so far: buffer = count & 1
        bool stuck = false;
        auto fetch = [&](int t) {
            if (lane == 0) tile_fetch(buf + (fetched & 1) * TILE4, rows + (int64_t)t * TILE4, TILE4 * 16, &bars[warp][fetched & 1]);
            ++fetched;
        };
        auto scan = [&]() {
            const uint32_t i = scanned & 1;
            stuck = !tile_wait(&bars[warp][i], (scanned >> 1) & 1);
            if (stuck) return;
            scan_tile<N, MODE>(reinterpret_cast<const ulonglong2*>(buf + i * TILE4), mm[0], mm[1], pv[0], pv[1]);
            ++scanned;
            __syncwarp();                                                      // read before it is fetched over
        };
        // ---- the tile nearest to one of the group's voxels ----
        float c[6], glo[6], ghi[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            c[k] = __shfl_sync(MADI_FULL, phi[0][k], 16);
            glo[k] = warp_minf32(fminf(phi[0][k], phi[1][k]));
            ghi[k] = warp_maxf32(fmaxf(phi[0][k], phi[1][k]));
        }
        float near = NO_SCORE;
        int t0 = 0;
        for (int t = lane; t < ix.n_tiles; t += 32) {
            const float d = box_distance2(boxes + 4ll * t, c, c);
            if (d < near) { near = d; t0 = t; }
        }
        {
            const float best = warp_minf32(near);
            const unsigned who = __ballot_sync(MADI_FULL, near == best);
            t0 = __shfl_sync(MADI_FULL, t0, who ? __ffs(who) - 1 : 0);
        }
        fetch(t0);
        scan();
        if (ix.test_stall && !tile_wait(&never, 0, STALL_POLLS)) stuck = true;
        // ---- every other tile some voxel still needs (this warp's share), one
        // in flight while the one before is scanned ----
        unsigned share = 0xffffffffu;
        if (WARPS > 1) share = (0x11111111u * ((1u << (4 / WARPS)) - 1u)) << (part * (4 / WARPS));
        for (int base = 0; base < ix.n_tiles && !stuck; base += 32) {
            const float top = warp_maxf32(fmaxf(pv[0].limit, pv[1].limit));
            const int mine = base + lane;
            bool want = false;
            if (mine < ix.n_tiles && mine != t0) want = !(0.998f * box_distance2(boxes + 4ll * mine, glo, ghi) > top);
            for (unsigned mask = __ballot_sync(MADI_FULL, want) & share; mask && !stuck; mask &= mask - 1) {
                const int t = base + __ffs(mask) - 1;
                const float4* b = boxes + 4ll * t;
                const bool need = !(0.998f * box_distance2(b, phi[0], phi[0]) > pv[0].limit) ||
                                  !(0.998f * box_distance2(b, phi[1], phi[1]) > pv[1].limit);
                if (!__any_sync(MADI_FULL, need)) continue;
                fetch(t);
                if (fetched - scanned == 2) scan();
            }
        }
        while (fetched != scanned && !stuck) scan();
        // a copy that did not complete in time (not seen; the waits are bounded): no
        // result is better than a wrong one.  The copies in flight are waited for
        // again, so that none lands in the next CTA's memory, and the call's status
        // says so (2: this wait ran out too).
        if (stuck) {
            pv[0].bj = pv[1].bj = -1;
            bool drained = true;
            for (; fetched != scanned; ++scanned) drained = tile_wait(&bars[warp][scanned & 1], (scanned >> 1) & 1) && drained;
            if (lane == 0) atomicMax(ix.status, drained ? 1 : 2);
        }
    }
    if (WARPS > 1) {
        const int g = warp / WARPS;
        if (live) {
#pragma unroll
            for (int i = 0; i < 2; ++i) atomicMin(&merged[g][32 * i + lane], pv[i].bj < 0 ? 0ull : match_key(pv[i].best, pv[i].bj));
        }
        __syncthreads();
        if (!live || part != 0) return;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const unsigned long long key = merged[g][32 * i + lane];
            pv[i].bj = key == 0ull ? -1 : (int)(uint32_t)key;
        }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
        if (p0 + 32 * i + lane < ix.n_vox) {
            if (pv[i].bj < 0) {
                best_idx[vox[i]] = -1;
                best_resid[vox[i]] = __int_as_float(0x7fc00000);
                if (MODE == MADI_MATCH_FREE_S0 && best_s0) best_s0[vox[i]] = __int_as_float(0x7fc00000);
            }
            else match_write<N, MODE>(meas, lib, vox[i], pv[i].bj, ix.F, best_idx, best_resid, best_s0);
        }
}

template <int N, int MODE, int WARPS>
static cudaError_t launch_pruned(const madi_match_desc* d, const prune::Index& ix, cudaStream_t s) {
    const auto kernel = match_pruned_kernel<N, MODE, WARPS>;
    constexpr int smem = MATCH_THREADS / 32 * 2 * prune::TILE * (N / 4 + 1) * 16;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    constexpr int per = 64 * (MATCH_THREADS / 32) / WARPS;
    kernel<<<(unsigned)((d->n_vox + per - 1) / per), MATCH_THREADS, smem, s>>>(d->measured, d->lib, ix, d->best_idx,
                                                                              d->best_resid, d->best_s0);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Which kernel (fp32)
// ---------------------------------------------------------------------------
struct MatchPlan {
    bool pruned;
    int parts;                  // library parts of the exhaustive scan
    int part;                   // entries a part
    int64_t bytes;              // scratch beyond the column means
};

static MatchPlan match_plan(int64_t n_vox, int32_t n_lib, int32_t n_feat) {
    MatchPlan p{false, 1, n_lib, 0};
    // The index costs ~0.1 ms: 20,000 voxels x 20,000 entries x 20 take 1.73 ms
    // scanned by one part, 0.20 ms pruned; 4,096 voxels 0.15 ms split over parts.
    if (n_vox >= 4096 && n_lib >= 1024 && n_lib <= prune::MAX_LIB && (double)n_vox * n_lib * n_feat >= 4e9 && n_vox < 0x7fffffff) {
        p.pruned = true;
        prune::Index ix;
        p.bytes = prune::layout(ix, nullptr, n_vox, n_lib, n_feat);
        return p;
    }
    // Small fits leave most SMs idle with one CTA per 128 voxels: about eight
    // CTAs an SM (1,216 of 152 SMs), a part no shorter than a chunk.  Two chunks are
    // not split: the memset and the second kernel cost what the shorter scan saves
    // (50 voxels x 200 entries x 5: 17.4 us in one part, 20.5 in two; 384 entries x
    // 20: 35 in one, 24 in three).
    const int64_t blocks = (n_vox + MATCH_THREADS - 1) / MATCH_THREADS;
    const int64_t chunks = ((int64_t)n_lib + MATCH_CHUNK - 1) / MATCH_CHUNK;
    const int64_t want = std::min<int64_t>(std::min<int64_t>(chunks, 65535), blocks > 0 ? 1216 / blocks : 1);
    if (want > 1 && chunks > 2) {
        p.part = (int)((chunks + want - 1) / want * MATCH_CHUNK);
        p.parts = (int)(((int64_t)n_lib + p.part - 1) / p.part);
        p.bytes = 8 * n_vox;
    }
    return p;
}

template <int N, int MODE>
static madi_status launch_fp32(const madi_match_desc* d, const MatchPlan& p, float* mu, unsigned char* scratch, cudaStream_t s) {
    if (p.pruned) {
        prune::Index ix;
        prune::layout(ix, scratch, d->n_vox, d->n_lib, d->n_feat);
        ix.mu = MODE == MADI_MATCH_FIXED_S0 ? mu : nullptr;
        ix.free_s0 = MODE == MADI_MATCH_FREE_S0;
        ix.test_stall = (d->flags & MADI_MATCH_FLAG_TEST_STALL) != 0;
        const madi_status st = prune::build(ix, d->measured, d->lib, true, s);
        if (st != MADI_OK) return st;
        // Warps a group: more shorten the longest group's chain of tiles while the
        // groups alone do not fill the chip, but each repeats the group's set-up and
        // holds a staler bound.  Fixed S0, 20,000 entries x 20, ms at 1 / 2 / 4 warps:
        // 50,000 voxels 0.40 / 0.29 / 0.24, 100,000 0.47 / 0.35 / 0.35, 125,000 0.49 /
        // 0.40 / 0.42, 200,000 0.59 / 0.54 / 0.60, 300,000 0.74 / 0.75 / 0.85, 1e6 2.02 /
        // 2.22 / 2.57.  40,000 entries, 10 or 28 features and free S0 cross over
        // within 75,000 to 150,000 and 200,000 to 400,000 voxels; the lines cost them
        // 10 % at most, and 8 % at 1,024 entries, where one warp is best from 200,000.
        const cudaError_t e = d->n_vox < 125000 ? launch_pruned<N, MODE, 4>(d, ix, s)
                              : d->n_vox < 300000 ? launch_pruned<N, MODE, 2>(d, ix, s)
                                                  : launch_pruned<N, MODE, 1>(d, ix, s);
        if (e != cudaSuccess) return host::cuda_fail(e, "match fp32 pruned launch");
    } else {
        unsigned long long* keys = p.parts > 1 ? reinterpret_cast<unsigned long long*>(scratch) : nullptr;
        if (keys) {
            const cudaError_t e = cudaMemsetAsync(keys, 0xff, 8 * d->n_vox, s);
            if (e != cudaSuccess) return host::cuda_fail(e, "match fp32 memset");
        }
        const int64_t blocks = (d->n_vox + MATCH_THREADS - 1) / MATCH_THREADS;
        // two voxels a thread halve the shared-memory reads; they pay from eight CTAs
        // an SM on (20,000 entries x 20, one / two: 200,000 voxels 6.4 / 4.7 ms, 80,000
        // 2.7 / 2.5, but free S0 3.1 / 3.8; 40,000 1.8 / 2.1)
        if (blocks >= 1216) {
            const dim3 grid((unsigned)((d->n_vox + 2 * MATCH_THREADS - 1) / (2 * MATCH_THREADS)), (unsigned)p.parts);
            match_scan_kernel<N, MODE, 2><<<grid, MATCH_THREADS, 0, s>>>(d->measured, d->lib, mu, d->n_vox, d->n_lib, d->n_feat,
                                                                        p.part, keys, d->best_idx, d->best_resid, d->best_s0);
        } else {
            match_scan_kernel<N, MODE, 1><<<dim3((unsigned)blocks, (unsigned)p.parts), MATCH_THREADS, 0, s>>>(
                d->measured, d->lib, mu, d->n_vox, d->n_lib, d->n_feat, p.part, keys, d->best_idx, d->best_resid, d->best_s0);
        }
        if (keys)
            match_finish_kernel<N, MODE><<<(unsigned)((d->n_vox + 255) / 256), 256, 0, s>>>(
                d->measured, d->lib, keys, d->n_vox, d->n_feat, d->best_idx, d->best_resid, d->best_s0);
    }
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return host::cuda_fail(e, "match fp32 launch");
    return MADI_OK;
}

template <int MODE>
static madi_status launch_fp32_mode(const madi_match_desc* d, const MatchPlan& p, float* mu, unsigned char* scratch, cudaStream_t s) {
    switch ((d->n_feat + 3) / 4) {
        case 1: case 2: return launch_fp32<8, MODE>(d, p, mu, scratch, s);
        case 3: return launch_fp32<12, MODE>(d, p, mu, scratch, s);
        case 4: return launch_fp32<16, MODE>(d, p, mu, scratch, s);
        case 5: return launch_fp32<20, MODE>(d, p, mu, scratch, s);
        case 6: return launch_fp32<24, MODE>(d, p, mu, scratch, s);
        case 7: return launch_fp32<28, MODE>(d, p, mu, scratch, s);
        default: return launch_fp32<32, MODE>(d, p, mu, scratch, s);
    }
}

}  // namespace madi

using namespace madi;

madi_status madi_match_bf16(const madi_match_desc* d, cudaStream_t s);
const int* madi_match_bf16_status_word(const madi_match_desc* d);
int64_t madi_match_bf16_scratch(int64_t n_vox, int32_t n_lib, int32_t n_feat, int32_t topk);
void madi_match_column_mean(const float* lib, int32_t n_lib, int32_t n_feat, float* mu, cudaStream_t s);

// fp32 needs room for the column means (fixed S0); with the plan's scratch behind
// them it splits or prunes the scan.
static constexpr int64_t FP32_SCRATCH = 256;

extern "C" int64_t madi_match_scratch_bytes(int64_t n_vox, int32_t n_lib, int32_t n_feat, int32_t precision,
                                            int32_t topk) {
    if (precision == MADI_MATCH_BF16) return madi_match_bf16_scratch(n_vox, n_lib, n_feat, topk);
    if (n_vox <= 0 || n_lib < 1 || n_feat < 1 || n_feat > 32) return FP32_SCRATCH;
    return FP32_SCRATCH + match_plan(n_vox, n_lib, n_feat).bytes;
}

// The route of an fp32 call and the scratch behind the column means it uses.
static MatchPlan fp32_route(const madi_match_desc* d, unsigned char*& scratch) {
    const MatchPlan plan = match_plan(d->n_vox, d->n_lib, d->n_feat);
    const bool ours = d->mode == MADI_MATCH_FIXED_S0 || (d->flags & MADI_MATCH_FLAG_SCRATCH);
    if (ours && d->scratch && (reinterpret_cast<uintptr_t>(d->scratch) & 255) == 0 &&
        d->scratch_bytes >= FP32_SCRATCH + plan.bytes) {
        scratch = static_cast<unsigned char*>(d->scratch) + FP32_SCRATCH;
        return plan;
    }
    return MatchPlan{false, 1, d->n_lib, 0};                // no scratch, or it holds the column means only
}

extern "C" madi_status madi_match(const madi_match_desc* d, void* stream) {
    host::clear_error();
    if (!d || !d->measured || !d->lib || !d->best_idx || !d->best_resid || d->n_vox < 0 || d->n_lib < 1 ||
        d->n_feat < 1)
        return host::fail(MADI_ERR_INVALID, "match: bad arguments");
    if (d->n_feat > 32) return host::fail(MADI_ERR_UNSUPPORTED, "match: at most 32 features");
    if (d->mode != MADI_MATCH_FIXED_S0 && d->mode != MADI_MATCH_FREE_S0)
        return host::fail(MADI_ERR_INVALID, "match: unknown mode");
    if (d->n_vox == 0) return MADI_OK;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (d->precision == MADI_MATCH_BF16) return madi_match_bf16(d, s);
    if (d->precision != MADI_MATCH_FP32) return host::fail(MADI_ERR_INVALID, "match: unknown precision");
    float* mu = nullptr;
    if (d->mode == MADI_MATCH_FIXED_S0) {
        if (!d->scratch || d->scratch_bytes < FP32_SCRATCH)
            return host::fail(MADI_ERR_CAPACITY, "match fp32: scratch %lld < %lld bytes", (long long)d->scratch_bytes,
                              (long long)FP32_SCRATCH);
        if ((reinterpret_cast<uintptr_t>(d->scratch) & 255) != 0)
            return host::fail(MADI_ERR_INVALID, "match fp32: scratch must be 256-byte aligned");
        mu = static_cast<float*>(d->scratch);
        madi_match_column_mean(d->lib, d->n_lib, d->n_feat, mu, s);
    }
    unsigned char* scratch = nullptr;
    const MatchPlan plan = fp32_route(d, scratch);
    return d->mode == MADI_MATCH_FIXED_S0 ? launch_fp32_mode<MADI_MATCH_FIXED_S0>(d, plan, mu, scratch, s)
                                          : launch_fp32_mode<MADI_MATCH_FREE_S0>(d, plan, mu, scratch, s);
}

extern "C" madi_status madi_match_wait(const madi_match_desc* d, void* stream) {
    host::clear_error();
    if (!d) return host::fail(MADI_ERR_INVALID, "match_wait: null descriptor");
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (d->precision == MADI_MATCH_FP32 && d->n_vox > 0 && d->n_lib > 0 && d->n_feat > 0 && d->n_feat <= 32) {
        unsigned char* scratch = nullptr;
        if (fp32_route(d, scratch).pruned) {
            prune::Index ix;
            prune::layout(ix, scratch, d->n_vox, d->n_lib, d->n_feat);
            int word = 0;
            cudaError_t e = cudaMemcpyAsync(&word, ix.status, sizeof(int), cudaMemcpyDeviceToHost, s);
            if (e == cudaSuccess) e = cudaStreamSynchronize(s);
            if (e != cudaSuccess) return host::cuda_fail(e, "match_wait: stream");
            if (word != 0)
                return host::fail(MADI_ERR_TIMEOUT, "match fp32: a bounded wait ran out; the voxels of the warps that gave up "
                                                    "have index -1 (%s)",
                                  word == 1 ? "issued copies were drained" : "and the drain of the issued copies ran out");
            return MADI_OK;
        }
    }
    cudaError_t e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return host::cuda_fail(e, "match_wait: stream");
    if (d->precision != MADI_MATCH_BF16 || d->n_vox == 0) return MADI_OK;
    if (!d->scratch || d->scratch_bytes < madi_match_bf16_scratch(d->n_vox, d->n_lib, d->n_feat, d->topk))
        return host::fail(MADI_ERR_INVALID, "match_wait: descriptor has no BF16 scratch");
    int word = 0;
    e = cudaMemcpyAsync(&word, madi_match_bf16_status_word(d), sizeof(int), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return host::cuda_fail(e, "match_wait: status word");
    if (word == 1)
        return host::fail(MADI_ERR_TIMEOUT, "match bf16: a bounded wait ran out; the rows of the CTAs that gave up "
                                            "have no result (issued copies and MMAs were drained)");
    if (word != 0)
        return host::fail(MADI_ERR_TIMEOUT, "match bf16: a bounded wait ran out and so did the drain of the issued "
                                            "copies and MMAs");
    return MADI_OK;
}
