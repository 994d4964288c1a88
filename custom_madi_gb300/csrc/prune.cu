// Construction of the pruned search's index (prune.cuh): directions, library
// order, tile rows and boxes, voxel order.  Every step but the counting sorts'
// scatter is deterministic; the order inside a bucket only moves which voxels
// share a warp and which entries share a tile, and no result depends on it.
#include "prune.cuh"

namespace madi {
namespace prune {

constexpr int BASIS_THREADS = 1024;
constexpr int ITERATIONS = 6;
constexpr int SROW = FMAX + 1;                  // sample row stride in shared memory (bank spread)

// Directions from a strided sample of the library: covariance, then orthogonal
// iteration.  One CTA; ranges of the projections of a library and a voxel sample.
__global__ void __launch_bounds__(BASIS_THREADS) basis_kernel(const float* __restrict__ meas, const float* __restrict__ lib,
                                                              const Index ix) {
    extern __shared__ float sm[];
    float* row = sm;                            // [SAMPLE][SROW]
    float* cov = sm + SAMPLE * SROW;            // [FMAX][FMAX]
    __shared__ float v[KDIR][FMAX], centre[FMAX];
    __shared__ int lo[6], hi[6];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int F = ix.F;
    auto load = [&](const float* x, int64_t n, int rows) {      // sampled rows, centred / scaled, into `row`
        if (tid < rows) {
            const float* r = x + ((int64_t)tid * n / rows) * F;
            float sc = 1.f;
            if (ix.free_s0) {
                float s = 0.f;
                for (int f = 0; f < F; ++f) s = fmaf(r[f], r[f], s);
                sc = s > 0.f ? rsqrtf(s) : 0.f;
            }
            for (int f = 0; f < F; ++f) row[tid * SROW + f] = ix.free_s0 ? r[f] * sc : r[f] - ix.mu[f];
        }
    };
    const int n = (int)min((int64_t)SAMPLE, (int64_t)ix.n_lib);
    load(lib, ix.n_lib, n);
    if (tid < FMAX) centre[tid] = 0.f;
    if (tid < 6) { lo[tid] = 0x7fffffff; hi[tid] = (int)0x80000000; }
    __syncthreads();
    if (ix.free_s0) {
        for (int f = warp; f < F; f += 32) {
            float s = 0.f;
            for (int i = lane; i < n; i += 32) s += row[i * SROW + f];
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(MADI_FULL, s, o);
            if (lane == 0) centre[f] = s / n;
        }
        __syncthreads();
        if (tid < n)
            for (int f = 0; f < F; ++f) row[tid * SROW + f] -= centre[f];
        __syncthreads();
    }
    for (int p = warp; p < FMAX * FMAX; p += 32) {
        const int a = p / FMAX, b = p % FMAX;
        if (a > b) continue;
        float s = 0.f;
        if (b < F)
            for (int i = lane; i < n; i += 32) s = fmaf(row[i * SROW + a], row[i * SROW + b], s);
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(MADI_FULL, s, o);
        if (lane == 0) cov[a * FMAX + b] = cov[b * FMAX + a] = s / n;
    }
    __syncthreads();
    if (warp == 0) {
        float x[KDIR];
#pragma unroll
        for (int k = 0; k < KDIR; ++k) x[k] = lane < F ? cosf(0.7f * (k + 1) * lane) + (lane == k ? 1.f : 0.f) : 0.f;
        for (int it = 0; it <= ITERATIONS; ++it) {
            if (it > 0) {
                float y[KDIR] = {};
                for (int b = 0; b < F; ++b) {
                    const float c = cov[lane * FMAX + b];
#pragma unroll
                    for (int k = 0; k < KDIR; ++k) y[k] = fmaf(c, __shfl_sync(MADI_FULL, x[k], b), y[k]);
                }
#pragma unroll
                for (int k = 0; k < KDIR; ++k) x[k] = y[k];
            }
            // Gram-Schmidt (each vector's sums together), twice in the last round; a
            // direction that vanishes becomes 0
            for (int rep = 0; rep < (it == ITERATIONS ? 2 : 1); ++rep) {
#pragma unroll
                for (int k = 0; k < KDIR; ++k) {
                    float d[KDIR];
#pragma unroll
                    for (int j = 0; j <= k; ++j) d[j] = x[k] * x[j];
                    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                        for (int j = 0; j <= k; ++j) d[j] += __shfl_xor_sync(MADI_FULL, d[j], o);
                    const float n0 = d[k];
#pragma unroll
                    for (int j = 0; j < k; ++j) x[k] = fmaf(-d[j], x[j], x[k]);
                    float n2 = x[k] * x[k];
                    for (int o = 16; o > 0; o >>= 1) n2 += __shfl_xor_sync(MADI_FULL, n2, o);
                    x[k] = (n2 > 1e-6f * n0 && n2 > 1e-30f) ? x[k] * (1.f / sqrtf(n2)) : 0.f;
                }
            }
        }
        for (int k = 0; k < KDIR; ++k) v[k][lane] = x[k];
    }
    __syncthreads();
    auto project = [&](int rows, int k0) {      // ranges of v_1..v_3 over the rows in shared memory
        float p[3] = {0.f, 0.f, 0.f};
        if (tid < rows)
            for (int f = 0; f < F; ++f)
                for (int k = 0; k < 3; ++k) p[k] = fmaf(row[tid * SROW + f], v[k][f], p[k]);
        for (int k = 0; k < 3; ++k) {
            const int o = f2o(p[k]);
            const int a = __reduce_min_sync(MADI_FULL, tid < rows ? o : 0x7fffffff);
            const int b = __reduce_max_sync(MADI_FULL, tid < rows ? o : (int)0x80000000);
            if (lane == 0) { atomicMin(&lo[k0 + k], a); atomicMax(&hi[k0 + k], b); }
        }
    };
    project(n, 0);
    __syncthreads();
    const int nv = (int)min((int64_t)SAMPLE, ix.n_vox);
    load(meas, ix.n_vox, nv);
    if (ix.free_s0 && tid < nv)
        for (int f = 0; f < F; ++f) row[tid * SROW + f] -= centre[f];
    __syncthreads();
    project(nv, 3);
    __syncthreads();
    for (int i = tid; i < KDIR * FMAX; i += BASIS_THREADS) ix.basis[i] = v[i / FMAX][i % FMAX];
    if (tid < FMAX) ix.basis[B_CENTRE + tid] = centre[tid];
    if (tid < 6) {
        ix.basis[B_RANGE + tid] = o2f(lo[tid]);
        ix.basis[B_RANGE + 6 + tid] = o2f(hi[tid]);
    }
}

// Bucket of p in [lo, hi] cut into n (NaN and values outside clamp).
MADI_DEV int bucket(float p, float lo, float hi, int n) {
    const float u = hi > lo ? (p - lo) / (hi - lo) * n : 0.f;
    return (int)fminf(fmaxf(u, 0.f), (float)(n - 1));
}

// One atomic per warp when every lane hits the same bin (masked-out voxels do).
MADI_DEV uint32_t bin_add(uint32_t* bins, uint32_t b) {
    const unsigned act = __activemask();
    int same;
    __match_all_sync(act, b, &same);
    if (!same) return atomicAdd(&bins[b], 1u);
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(act) - 1;
    uint32_t base = 0;
    if (lane == leader) base = atomicAdd(&bins[b], (uint32_t)__popc(act));
    return __shfl_sync(act, base, leader) + __popc(act & ((1u << lane) - 1u));
}

// Embeds and bins the library (first blocks) and the voxels (the rest).
template <int N>
__global__ void __launch_bounds__(256) embed_kernel(const float* __restrict__ meas, const float* __restrict__ lib,
                                                    const Index ix, int lib_blocks) {
    __shared__ float sv[B_FLOATS], smu[FMAX];
    for (int i = threadIdx.x; i < B_FLOATS; i += 256) sv[i] = ix.basis[i];
    if (threadIdx.x < FMAX) smu[threadIdx.x] = (ix.mu && (int)threadIdx.x < ix.F) ? ix.mu[threadIdx.x] : 0.f;
    __syncthreads();
    const bool is_lib = (int)blockIdx.x < lib_blocks;
    const int64_t i = (int64_t)(is_lib ? blockIdx.x : blockIdx.x - lib_blocks) * 256 + threadIdx.x;
    const int64_t n = is_lib ? ix.n_lib : ix.n_vox;
    if (i >= n) return;
    const float* r = (is_lib ? lib : meas) + i * ix.F;
    float x[N];
    float n2 = 0.f;
#pragma unroll
    for (int f = 0; f < N; ++f) {
        x[f] = f < ix.F ? r[f] - smu[f] : 0.f;
        n2 = fmaf(x[f], x[f], n2);
    }
    if (ix.free_s0) {
        const float sc = n2 > 0.f ? rsqrtf(n2) : 0.f;
#pragma unroll
        for (int f = 0; f < N; ++f) x[f] = f < ix.F ? fmaf(x[f], sc, -sv[B_CENTRE + f]) : 0.f;
    }
    const float* rg = sv + B_RANGE;             // low: library 3, voxels 3; high: the same
    if (is_lib) {
        const Phi e = embed(x, sv);
        float4* o = reinterpret_cast<float4*>(ix.phi + 8 * i);
        o[0] = make_float4(e.p[0], e.p[1], e.p[2], e.p[3]);
        o[1] = make_float4(e.p[4], e.q, 0.f, 0.f);
        // non-negative floats order as their bits; NaN orders above all of them
        atomicMax(reinterpret_cast<int*>(ix.lmax), __float_as_int(fabsf(n2 * 1.00001f)));
        if (ix.free_s0 && n2 > 0.f) atomicMax(reinterpret_cast<int*>(ix.lmax) + 1, __float_as_int(1.f / fmaxf(n2, 1e-30f)));
        const int a = bucket(e.p[0], rg[0], rg[6], ix.slabs);
        int b = bucket(e.p[1], rg[1], rg[7], LIB_FINE);
        if (a & 1) b = LIB_FINE - 1 - b;        // neighbouring slabs meet at the same end
        ix.lbin[i] = (uint32_t)(a * LIB_FINE + b);
        bin_add(ix.bins, ix.lbin[i]);
    } else {
        float p[3] = {0.f, 0.f, 0.f};
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int f = 0; f < N; ++f) p[k] = fmaf(x[f], sv[k * FMAX + f], p[k]);
        const int a = bucket(p[0], rg[3], rg[9], 64), b = bucket(p[1], rg[4], rg[10], 32), c = bucket(p[2], rg[5], rg[11], 16);
        const uint32_t key = (uint32_t)((a * 32 + ((a & 1) ? 31 - b : b)) * 16 + ((b & 1) ? 15 - c : c));
        ix.vbin[i] = key;
        bin_add(ix.bins + LIB_BINS, key);
    }
}

// Exclusive scan of the bins: CTA 0 the library's, CTA 1 the voxels'.  A warp
// takes a contiguous 32nd, 128 bins per coalesced step.
__global__ void __launch_bounds__(1024) scan_kernel(uint32_t* bins) {
    static_assert(LIB_BINS % 4096 == 0 && VOX_BINS % 4096 == 0, "whole steps");
    constexpr int MAX_STEPS = (LIB_BINS > VOX_BINS ? LIB_BINS : VOX_BINS) / 4096;
    __shared__ uint32_t part[32];
    uint32_t* b = blockIdx.x == 0 ? bins : bins + LIB_BINS;
    const int steps = (blockIdx.x == 0 ? LIB_BINS : VOX_BINS) / 4096;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint4* mine = reinterpret_cast<uint4*>(b) + warp * steps * 32 + lane;
    uint4 x[MAX_STEPS];
    uint32_t sum = 0;
#pragma unroll
    for (int i = 0; i < MAX_STEPS; ++i)
        if (i < steps) x[i] = mine[32 * i];
#pragma unroll
    for (int i = 0; i < MAX_STEPS; ++i)
        if (i < steps) sum += x[i].x + x[i].y + x[i].z + x[i].w;
    sum = __reduce_add_sync(MADI_FULL, sum);
    if (lane == 0) part[warp] = sum;
    __syncthreads();
    uint32_t run = __reduce_add_sync(MADI_FULL, lane < warp ? part[lane] : 0u);
#pragma unroll
    for (int i = 0; i < MAX_STEPS; ++i) {
        if (i >= steps) break;
        const uint32_t s4 = x[i].x + x[i].y + x[i].z + x[i].w;
        uint32_t inc = s4;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t u = __shfl_up_sync(MADI_FULL, inc, o);
            if (lane >= o) inc += u;
        }
        uint4 y;
        y.x = run + inc - s4; y.y = y.x + x[i].x; y.z = y.y + x[i].y; y.w = y.z + x[i].z;
        mine[32 * i] = y;
        run += __shfl_sync(MADI_FULL, inc, 31);
    }
}

__global__ void __launch_bounds__(256) scatter_kernel(const Index ix, int lib_blocks) {
    const bool is_lib = (int)blockIdx.x < lib_blocks;
    const int64_t i = (int64_t)(is_lib ? blockIdx.x : blockIdx.x - lib_blocks) * 256 + threadIdx.x;
    if (is_lib) {
        if (i < ix.n_lib) ix.lperm[bin_add(ix.bins, ix.lbin[i])] = (int32_t)i;
        else if (i < (int64_t)ix.n_tiles * TILE) ix.lperm[i] = -1;
    } else if (i < ix.n_vox) {
        ix.vperm[bin_add(ix.bins + LIB_BINS, ix.vbin[i])] = (int32_t)i;
    }
}

// One CTA per tile: entries in ascending index order, rows (fixed S0: centred),
// |row|^2 as the exhaustive scan computes it, and the box of their Phi.
__global__ void __launch_bounds__(TILE) tile_kernel(const float* __restrict__ lib, const Index ix) {
    __shared__ int idx[TILE], sorted[TILE];
    __shared__ float red[2][6][TILE / 32];
    const int t = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int e = ix.lperm[t * TILE + tid];
    const int key = e < 0 ? 0x7fffffff : e;
    idx[tid] = key;
    __syncthreads();
    int rank = 0;
    for (int i = 0; i < TILE; ++i) rank += idx[i] < key || (idx[i] == key && i < tid);
    sorted[rank] = e;
    __syncthreads();
    const int j = sorted[tid];
    ix.lperm[t * TILE + tid] = j;
    // pairs of entries, feature by feature: (x_0[f], x_1[f]), then (|x_0|^2, |x_1|^2,
    // index, index)
    const int w = ix.stride - 4, half = tid & 1;
    float* out = ix.rows + (int64_t)(t * (TILE / 2) + (tid >> 1)) * (2 * ix.stride);
    float s = 0.f;
    for (int f = 0; f < w; ++f) {
        const float x = (j >= 0 && f < ix.F) ? lib[(int64_t)j * ix.F + f] - (ix.mu ? ix.mu[f] : 0.f) : 0.f;
        s = fmaf(x, x, s);
        out[2 * f + half] = x;
    }
    // padding entries score NaN (free S0: no positive dot product) and never win
    out[2 * w + half] = j >= 0 ? (ix.free_s0 ? fmaxf(s, 1e-30f) : s) : __int_as_float(0x7fc00000);
    out[2 * w + 2 + half] = __int_as_float(j);
    out[2 * w + 4 + half] = out[2 * w + 6 + half] = 0.f;
    for (int k = 0; k < 6; ++k) {
        float lo = j >= 0 ? ix.phi[8ll * j + k] : 3.0e38f, hi = j >= 0 ? lo : -3.0e38f;
        for (int o = 16; o > 0; o >>= 1) {
            lo = fminf(lo, __shfl_xor_sync(MADI_FULL, lo, o));
            hi = fmaxf(hi, __shfl_xor_sync(MADI_FULL, hi, o));
        }
        if (lane == 0) { red[0][k][warp] = lo; red[1][k][warp] = hi; }
    }
    __syncthreads();
    if (tid < 6) {
        float lo = red[0][tid][0], hi = red[1][tid][0];
        for (int w = 1; w < TILE / 32; ++w) { lo = fminf(lo, red[0][tid][w]); hi = fmaxf(hi, red[1][tid][w]); }
        ix.box[16ll * t + tid] = lo;
        ix.box[16ll * t + 8 + tid] = hi;
    }
}

template <int N>
static void launch_embed(const Index& ix, const float* meas, const float* lib, int lib_blocks, int vox_blocks, cudaStream_t s) {
    embed_kernel<N><<<lib_blocks + vox_blocks, 256, 0, s>>>(meas, lib, ix, lib_blocks);
}

madi_status build(const Index& ix, const float* meas, const float* lib, bool tiles, cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(ix.bins, 0, (LIB_BINS + VOX_BINS) * 4 + 256, s);
    if (e != cudaSuccess) return host::cuda_fail(e, "search index memset");
    constexpr int smem = (SAMPLE * SROW + FMAX * FMAX) * 4;
    e = cudaFuncSetAttribute(basis_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return host::cuda_fail(e, "search index attribute");
    basis_kernel<<<1, BASIS_THREADS, smem, s>>>(meas, lib, ix);
    const int lib_blocks = (ix.n_tiles * TILE + 255) / 256;
    const int vox_blocks = (int)((ix.n_vox + 255) / 256);
    if (ix.F <= 8) launch_embed<8>(ix, meas, lib, lib_blocks, vox_blocks, s);
    else if (ix.F <= 16) launch_embed<16>(ix, meas, lib, lib_blocks, vox_blocks, s);
    else if (ix.F <= 24) launch_embed<24>(ix, meas, lib, lib_blocks, vox_blocks, s);
    else launch_embed<32>(ix, meas, lib, lib_blocks, vox_blocks, s);
    scan_kernel<<<2, 1024, 0, s>>>(ix.bins);
    const int sort_blocks = tiles ? lib_blocks : 0;
    scatter_kernel<<<sort_blocks + vox_blocks, 256, 0, s>>>(ix, sort_blocks);
    if (tiles) tile_kernel<<<ix.n_tiles, TILE, 0, s>>>(lib, ix);
    e = cudaGetLastError();
    if (e != cudaSuccess) return host::cuda_fail(e, "search index launch");
    return MADI_OK;
}

}  // namespace prune
}  // namespace madi
