// Bayesian posterior-mean fit over the library, replacing _bayes_kernel_fixed /
// _bayes_kernel_free_s0 (madi/fitters_gpu.py:156-294) and the CPU bayes_fit
// (madi/fitters.py:110-243).
//
// Per voxel, library entry j gets log-weight e_j = log q_j - rw_j / (2 sigma^2)
// with q_j the quadrature weight and rw_j the residual on the normalised scale
// (fixed S0: |m - L_j|^2; free S0: |m/s0_j - L_j|^2, s0_j = m.L_j / |L_j|^2 > 0,
// other entries weight 0).  Outputs are the posterior means and standard
// deviations of (kio, rho, V), the weighted residual, n_eff = W^2 / sum w^2 and
// (free S0) the weighted S0.
//
// One voxel per lane, the library in index order, twice:
//   pass 1: the fp32 scores of the entries (the match kernel's centred fixed-S0
//           score, or the free-S0 projection), argmax of e_j -> j*; e_j* is then
//           recomputed from the direct difference and is the shift S (the
//           reference shifts by the minimum residual or the maximum log-weight;
//           any shift gives the same normalised weights).
//   pass 2: entries that can be above S - CUT get the direct-difference residual
//           (error ~F ulp of the residual itself, which is small where weights
//           matter); those that are above it add
//           w = exp(e_j - S) to Kahan-compensated fp32 sums of w, w d, w d^2
//           (d = parameter minus that of j*, so narrow posteriors keep their
//           variance), w r, w^2 and w s0.  Entries below the cut weigh less
//           than e^-CUT of entry j*.
//
// Most of the time went into fp64: d took three fp64 subtractions and conversions
// per (warp, entry) that passed, at two fp64 lanes per SM and cycle, and with
// voxels in file order nearly every entry passed for some lane.  Here
//   - voxels are taken in the order of the search index (prune.cuh), so that the
//     32 voxels of a warp need the same entries;
//   - a warp tests 32 entries at a time, one per lane, against the box of its
//     voxels in the index's embedding and only visits those that can matter;
//   - d is formed from three floats a parameter, which hold its 53 bits, and
//     rounded to fp32 once as before.
// The entries a voxel sums, and their order, are unchanged.  100,000 voxels x
// 20,000 entries x 20 features, sigma_m 0.02: 33.2 ms before, 7.0 ms now (5.9 ms of it this
// kernel, bound by issue; the rest is the index and host copies).
#include <cstdint>
#include "madi_device.cuh"
#include "madi_host.h"
#include "prune.cuh"

namespace madi {
namespace bayes {

constexpr int CHUNK = 128;           // entries staged at a time
constexpr float CUT = 60.f;          // exp(-60) ~ 9e-27 of the shift entry's weight

// Two compensated sums of products in packed registers.  y = a b - c is one fused
// operation; c is kept negated.
struct Kahan2 {
    uint64_t s = 0, nc = 0;
    MADI_DEV void add(uint64_t a, uint64_t b) {
        const uint64_t y = fma2(a, b, nc);
        const uint64_t t = add2(s, y);
        nc = sub2(y, sub2(t, s));
        s = t;
    }
    MADI_DEV void scale(uint64_t f) { s = mul2(s, f); nc = mul2(nc, f); }
    MADI_DEV double lo() const { return (double)split2(s).x + (double)split2(nc).x; }
    MADI_DEV double hi() const { return (double)split2(s).y + (double)split2(nc).y; }
};

struct Plan {
    const float* meas;
    const float* lib;
    const float* mu;                 // column means (fixed S0), zeros (free S0)
    const double* logq;
    const double* kio;
    const double* rho;
    const double* V;
    int64_t n_vox;
    int n_lib, F;
    float inv2s2;
    double* out;
    prune::Index ix;                 // indexed plans only
    float* blocks;                   // [n_lib][Entry floats], indexed plans only
};

// One entry in shared memory: centred (fixed S0) or raw (free S0) row, raw row,
// then |row|^2, log q, and kio, rho, V in three parts each: (kio, rho) high, middle,
// low, V high, middle, low, 1 if one of them is not in parts (else 0).
template <int N>
struct Entry {
    static constexpr int RAW = N, AUX = 2 * N, FLOATS = 2 * N + 12;
};

// x = h + m + l exactly: h to 24 bits, m a multiple of 2^-46 of h's binade (so that
// differences of two middles are exact wherever the highs are near each other), l the
// rest, <= 7 bits.  `out`: x is outside the range where all three are exact.
struct Parts { float h, m, l; };
MADI_DEV Parts parts_of(double x, bool& out) {
    const float h = (float)x;
    if (!(fabsf(h) >= 1e-28f && fabsf(h) <= 3.4e38f)) {
        out |= x != 0.0;
        return Parts{0.f, 0.f, 0.f};
    }
    const double r = x - (double)h;
    const float grid = __int_as_float(((__float_as_int(h) & 0x7f800000) - (23 << 23)) | 0x400000);       // 1.5 2^(E - 23)
    const float m = __fadd_rn(__fadd_rn((float)r, grid), -grid);
    return Parts{h, m, (float)(r - (double)m)};
}

// Differences a - b of two values at a time, rounded to fp32 once: where the highs
// are near, s, m, l and s + m are exact; elsewhere e and g are the errors of s and p.
// (Two floats a value hold 48 bits: for parameters that agree to 2^-25 the
// difference was short of bits.  100,000 voxels x 20,000 entries x 20: 6.4 ms a fit
// with two, 7.0 ms with three.)
MADI_DEV uint64_t parts_diff(uint64_t ah, uint64_t am, uint64_t al, uint64_t bh, uint64_t bm, uint64_t bl) {
    const uint64_t s = sub2(ah, bh);
    const uint64_t t = sub2(s, ah);
    const uint64_t e = sub2(sub2(ah, sub2(s, t)), add2(bh, t));
    const uint64_t m = sub2(am, bm);
    const uint64_t p = add2(s, m);
    const uint64_t g = sub2(m, sub2(p, s));
    return add2(p, add2(add2(e, g), sub2(al, bl)));
}

// The same in fp64, from memory; a call of its own so that nothing of it is done ahead.
__device__ __noinline__ float diff_f64(const double* a, double b) { return (float)(*a - b); }

// Screened log-weight of one entry from the fp32 score.
template <int FMAX, bool FREE>
MADI_DEV float screen(const float* m, const float* l, float sn, float lq, float m2, float inv2s2) {
    float dot = 0.f;
#pragma unroll
    for (int f = 0; f < FMAX; ++f) dot = fmaf(m[f], l[f], dot);
    if (!FREE) {
        // centred: r = |m~|^2 + |L~|^2 - 2 m~.L~ ; fp32 error <= (F + 4) 2^-23 (|m~|^2 + |L~|^2)
        const float r = fmaxf(fmaf(-2.f, dot, sn) + m2, 0.f);
        return lq - r * inv2s2;
    }
    // rw = |L|^2 (|m|^2 |L|^2 / (m.L)^2 - 1) when m.L > 0
    if (!(dot > 0.f)) return -3.0e38f;
    const float ratio = m2 * sn / (dot * dot);
    const float rw = fmaxf(sn * (ratio - 1.f), 0.f);
    return lq - rw * inv2s2;
}

// Residuals of one entry from the direct difference (raw data): resid (the
// reported residual) and rw (normalised), s0 (free S0; 1 for fixed).
template <int FMAX, bool FREE>
MADI_DEV bool exact(const float* mr, const float* L, int F, float& resid, float& rw, float& s0) {
    s0 = 1.f;
    if (FREE) {
        float dot = 0.f, rr = 0.f;
#pragma unroll
        for (int f = 0; f < FMAX; ++f) {
            if (f < F) { dot = fmaf(mr[f], L[f], dot); rr = fmaf(L[f], L[f], rr); }
        }
        if (!(dot > 0.f)) return false;
        s0 = dot / fmaxf(rr, 1e-30f);
    }
    float r = 0.f;
#pragma unroll
    for (int f = 0; f < FMAX; ++f) {
        if (f < F) {
            const float d = mr[f] - s0 * L[f];
            r = fmaf(d, d, r);
        }
    }
    resid = r;
    rw = FREE ? r / (s0 * s0) : r;
    return true;
}

// The same for an entry of the staged form (zero padded rows; |L|^2 as staged),
// two differences at a time, summed in the same order.
template <int N, bool FREE>
MADI_DEV bool exact_staged(const float* mr, const uint64_t* mr2, const float* o, float& resid, float& rw, float& s0) {
    const ulonglong2* L2 = reinterpret_cast<const ulonglong2*>(o + Entry<N>::RAW);
    float dot = 0.f;
    s0 = 1.f;
    if (FREE) {
        const float4* L = reinterpret_cast<const float4*>(o + Entry<N>::RAW);
#pragma unroll
        for (int f = 0; f < N / 4; ++f) {
            const float4 l = L[f];
            dot = fmaf(mr[4 * f], l.x, dot); dot = fmaf(mr[4 * f + 1], l.y, dot);
            dot = fmaf(mr[4 * f + 2], l.z, dot); dot = fmaf(mr[4 * f + 3], l.w, dot);
        }
        s0 = dot / o[Entry<N>::AUX];
    }
    const uint64_t ms0 = pair2(-s0, -s0);
    float r = 0.f;
#pragma unroll
    for (int f = 0; f < N / 4; ++f) {
        const ulonglong2 l = L2[f];
        const float2 a = split2(fma2(l.x, ms0, mr2[2 * f])), b = split2(fma2(l.y, ms0, mr2[2 * f + 1]));
        r = fmaf(a.x, a.x, r); r = fmaf(a.y, a.y, r);
        r = fmaf(b.x, b.x, r); r = fmaf(b.y, b.y, r);
    }
    resid = r;
    rw = FREE ? r / (s0 * s0) : r;
    return !FREE || dot > 0.f;
}

// Entry e of the library in the staged form.
template <int N, bool FREE>
MADI_DEV void make_entry(const Plan& P, int64_t e, const float* smu, float* o) {
    float sn = 0.f;
    for (int f = 0; f < N; ++f) {
        const float x = f < P.F ? P.lib[e * P.F + f] : 0.f;
        const float c = f < P.F ? x - smu[f] : 0.f;
        o[f] = c;
        o[Entry<N>::RAW + f] = x;
        sn = fmaf(c, c, sn);
    }
    float* a = o + Entry<N>::AUX;
    a[0] = FREE ? fmaxf(sn, 1e-30f) : sn;
    a[1] = (float)P.logq[e];
    bool out = false;
    const Parts k = parts_of(P.kio[e], out), r = parts_of(P.rho[e], out), v = parts_of(P.V[e], out);
    a[2] = k.h; a[3] = r.h; a[4] = k.m; a[5] = r.m; a[6] = k.l; a[7] = r.l;
    a[8] = v.h; a[9] = v.m; a[10] = v.l; a[11] = out ? 1.f : 0.f;
}

// The library in the staged form, and (|row|^2, log q) beside its embedding.
template <int N, bool FREE>
__global__ void __launch_bounds__(128) bayes_prep_kernel(const Plan P) {
    __shared__ float smu[N];
    if (threadIdx.x < N) smu[threadIdx.x] = (!FREE && (int)threadIdx.x < P.F) ? P.mu[threadIdx.x] : 0.f;
    __syncthreads();
    const int64_t e = (int64_t)blockIdx.x * 128 + threadIdx.x;
    if (e >= P.n_lib) return;
    float* o = P.blocks + e * Entry<N>::FLOATS;
    make_entry<N, FREE>(P, e, smu, o);
    P.ix.phi[8 * e + 6] = o[Entry<N>::AUX];
    P.ix.phi[8 * e + 7] = o[Entry<N>::AUX + 1];
}

// Largest of a warp's values (no NaN).
MADI_DEV float warp_maxf_bits(float v) { return o2f(__reduce_max_sync(MADI_FULL, f2o(v))); }

// Least residual rw an entry with embedding distance^2 d2 and |row|^2 sn can
// have, and more than the screen and its error bound are off, in rw units.
// Fixed S0: d2 >= |m - L|^2 bounds from below, fp32 scores are off by at most e
// (see match_pruned_kernel).  Free S0: cos <= 1 - d2 / 2 and rw = sn (1 / cos^2 - 1).
template <bool FREE>
MADI_DEV float least_rw(float d2, float sn, float e) {
    if (!FREE) return 0.998f * d2 - e;
    const float c = fmaxf(1.f - 0.499f * d2, 0.05f);
    return sn * ((1.f / (c * c) - 1.f) * 0.998f - 1e-4f);
}

template <int N, bool FREE, int THREADS, bool INDEXED>
__global__ void __launch_bounds__(THREADS) bayes_kernel(const __grid_constant__ Plan P) {
    constexpr int EF = Entry<N>::FLOATS;
    extern __shared__ __align__(16) float sent[];            // [CHUNK][EF]
    __shared__ float smu[N], sv[INDEXED ? prune::B_FLOATS : 1];
    const int F = P.F, lane = threadIdx.x & 31;
    const int64_t slot = (int64_t)blockIdx.x * THREADS + threadIdx.x;
    const bool live = slot < P.n_vox;
    const int64_t v = INDEXED ? (int64_t)P.ix.vperm[min(slot, P.n_vox - 1)] : min(slot, P.n_vox - 1);
    if (threadIdx.x < N) smu[threadIdx.x] = (!FREE && (int)threadIdx.x < F) ? P.mu[threadIdx.x] : 0.f;
    if (INDEXED)
        for (int i = threadIdx.x; i < prune::B_FLOATS; i += THREADS) sv[i] = P.ix.basis[i];
    __syncthreads();
    float m[N], mr[N];
    float m2 = 0.f;
#pragma unroll
    for (int f = 0; f < N; ++f) {
        mr[f] = f < F ? P.meas[v * F + f] : 0.f;
        m[f] = f < F ? mr[f] - smu[f] : 0.f;
        m2 = fmaf(m[f], m[f], m2);
    }
    // box of the warp's voxels in the embedding; e: margin on a residual (fixed S0)
    float glo[6], ghi[6], e_max = 0.f;
    bool bounded = false;
    if (INDEXED) {
        prune::Phi ph;
        if (!FREE) {
            ph = prune::embed(m, sv);
        } else {
            float u[N];
            const float sc = m2 > 0.f ? rsqrtf(m2) : 0.f;
#pragma unroll
            for (int f = 0; f < N; ++f) u[f] = f < F ? fmaf(m[f], sc, -sv[prune::B_CENTRE + f]) : 0.f;
            ph = prune::embed(u, sv);
        }
        const float lmax = P.ix.lmax[0];
        const bool ok = FREE ? m2 < 1e30f && m2 * lmax < 1e30f && m2 > 1e-25f * P.ix.lmax[1] && P.ix.lmax[1] < 1e20f
                             : m2 + lmax < 1e30f && m2 + lmax > 1e-30f;
        bounded = __all_sync(MADI_FULL, ok);
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            const float x = k < 5 ? ph.p[k] : ph.q;
            glo[k] = o2f(__reduce_min_sync(MADI_FULL, f2o(x)));
            ghi[k] = o2f(__reduce_max_sync(MADI_FULL, f2o(x)));
        }
        // screen error (F + 8) 2^-21 (|m|^2 + |L|^2) twice, and the bound added to it
        e_max = warp_maxf_bits((float)((N + 7) / 8 * 8 + 8) * 2e-6f * (m2 + lmax));
    }
    // Visits, in index order and by twos, the entries that may reach `floor` (a
    // log-weight) for some voxel of the warp; visit runs warp-wide.
    auto sweep = [&](auto floor, auto visit) {
        for (int base = 0; base < P.n_lib; base += CHUNK) {
            const int cnt = min(CHUNK, P.n_lib - base);
            unsigned mask[CHUNK / 32];
            unsigned any = 0;
            const float lim = floor();
#pragma unroll
            for (int i = 0; i < CHUNK / 32; ++i) {
                const int k = 32 * i + lane;
                bool want = k < cnt;
                if (INDEXED && bounded && want) {
                    const float4* q = reinterpret_cast<const float4*>(P.ix.phi + 8 * (int64_t)(base + k));
                    const float4 a = q[0], b = q[1];
                    const float x[6] = {a.x, a.y, a.z, a.w, b.x, b.y};
                    float d2 = 0.f;
#pragma unroll
                    for (int j = 0; j < 6; ++j) {
                        const float d = fmaxf(fmaxf(x[j] - ghi[j], glo[j] - x[j]), 0.f);
                        d2 = fmaf(d, d, d2);
                    }
                    want = !(b.w - least_rw<FREE>(d2, b.z, e_max) * P.inv2s2 + 3e-3f < lim);
                }
                mask[i] = __ballot_sync(MADI_FULL, want);
                any |= mask[i];
            }
            if (THREADS > 32 ? !__syncthreads_or(any != 0u) : any == 0u) continue;
            if (THREADS == 32) __syncwarp();
            if (INDEXED) {
                const float4* src = reinterpret_cast<const float4*>(P.blocks + (int64_t)base * EF);
                float4* dst = reinterpret_cast<float4*>(sent);
                for (int t = threadIdx.x; t < cnt * (EF / 4); t += THREADS) dst[t] = src[t];
            } else {
                for (int t = threadIdx.x; t < cnt; t += THREADS) make_entry<N, FREE>(P, base + t, smu, sent + t * EF);
            }
            if (THREADS > 32) __syncthreads(); else __syncwarp();
#pragma unroll
            for (int i = 0; i < CHUNK / 32; ++i)
                for (unsigned w = mask[i]; w;) {
                    // two entries at a time: their residuals are independent chains
                    const int k0 = 32 * i + __ffs(w) - 1;
                    w &= w - 1;
                    const bool two = w != 0u;
                    const int k1 = two ? 32 * i + __ffs(w) - 1 : k0;
                    w &= w - 1;
                    visit(base + k0, sent + k0 * EF, base + k1, sent + k1 * EF, two);
                }
            if (THREADS > 32) __syncthreads(); else __syncwarp();
        }
    };
    // ---- pass 1: argmax of the screened log-weight ----
    float best = -3.0e38f;
    int bj = -1;
    float known = -3.0e38f;                                  // a log-weight every voxel of the warp reaches
    if (INDEXED && bounded) {
        // the screened weight of the entry that looks best for one of the voxels
        float c[6], top = -3.0e38f;
#pragma unroll
        for (int k = 0; k < 6; ++k) c[k] = 0.5f * (glo[k] + ghi[k]);
        int tj = 0;
        for (int e = lane; e < P.n_lib; e += 32) {
            const float4* q = reinterpret_cast<const float4*>(P.ix.phi + 8 * (int64_t)e);
            const float4 a = q[0], b = q[1];
            const float x[6] = {a.x, a.y, a.z, a.w, b.x, b.y};
            float d2 = 0.f;
#pragma unroll
            for (int j = 0; j < 6; ++j) d2 = fmaf(x[j] - c[j], x[j] - c[j], d2);
            const float u = b.w - least_rw<FREE>(d2, b.z, 0.f) * P.inv2s2;
            if (u > top) { top = u; tj = e; }
        }
        const float w = warp_maxf_bits(top);
        const unsigned who = __ballot_sync(MADI_FULL, top == w);
        tj = __shfl_sync(MADI_FULL, tj, who ? __ffs(who) - 1 : 0);
        const float* o = P.blocks + (int64_t)tj * EF;
        known = screen<N, FREE>(m, o, o[Entry<N>::AUX], o[Entry<N>::AUX + 1], m2, P.inv2s2);
    }
    sweep([&]() { return warp_minf(fmaxf(best, known)); },
          [&](int e0, const float* o0, int e1, const float* o1, bool two) {
              const float ee0 = screen<N, FREE>(m, o0, o0[Entry<N>::AUX], o0[Entry<N>::AUX + 1], m2, P.inv2s2);
              const float ee1 = screen<N, FREE>(m, o1, o1[Entry<N>::AUX], o1[Entry<N>::AUX + 1], m2, P.inv2s2);
              if (ee0 > best) { best = ee0; bj = e0; }
              if (two && ee1 > best) { best = ee1; bj = e1; }
          });
    // shift and centre from the exact residual of j*
    float S = 0.f;
    double x0[3] = {0.0, 0.0, 0.0};
    uint64_t xh = 0, xm = 0, xl = 0;                         // parts of (kio, rho) of j*
    Parts xv{0.f, 0.f, 0.f};                                 // and of its V
    bool x_out = false;
    bool any = bj >= 0;
    if (any) {
        float Lj[N];
#pragma unroll
        for (int f = 0; f < N; ++f) Lj[f] = f < F ? P.lib[(int64_t)bj * F + f] : 0.f;
        float resid, rw, s0;
        any = exact<N, FREE>(mr, Lj, F, resid, rw, s0);
        S = (float)P.logq[bj] - rw * P.inv2s2;
        x0[0] = P.kio[bj];
        x0[1] = P.rho[bj];
        x0[2] = P.V[bj];
        const Parts k = parts_of(x0[0], x_out), r = parts_of(x0[1], x_out);
        xh = pair2(k.h, r.h);
        xm = pair2(k.m, r.m);
        xl = pair2(k.l, r.l);
        xv = parts_of(x0[2], x_out);
    }
    // ---- pass 2: exp-weighted sums over the entries above the cut ----
    // Sums in pairs: (w, w^2), (w resid, w s0), (w d_kio, w d_rho), (w d_V, w d_V^2),
    // (w d_kio^2, w d_rho^2).  Entries the sweep visits go to the exact residual at
    // once: most pass, and the cut on the exact log-weight is the one that counts.
    Kahan2 WW, RS, D1, DV, D2;
    uint64_t mr2[N / 2];
#pragma unroll
    for (int f = 0; f < N / 2; ++f) mr2[f] = pair2(mr[2 * f], mr[2 * f + 1]);
    sweep([&]() {
              // entries below S - CUT of every voxel; a voxel without any entry sums none
              const float s = warp_minf(any ? S : 3.0e38f);
              return s - CUT - 1e-5f * fabsf(s);
          },
          [&](int e0, const float* o0, int e1, const float* o1, bool two) {
              float resid0, rw0, s00, resid1, rw1, s01;
              const bool fits0 = exact_staged<N, FREE>(mr, mr2, o0, resid0, rw0, s00) && any;
              const bool fits1 = exact_staged<N, FREE>(mr, mr2, o1, resid1, rw1, s01) && any && two;
              auto add = [&](int entry, const float* a, float resid, float rw, float s0) {
                  float x = a[1] - rw * P.inv2s2 - S;
                  if (!(x > -CUT)) return;
                  if (x > 0.f) {
                      // an entry above the screened maximum (within the screen's error):
                      // move the shift to it so that every weight stays <= 1
                      const float f = expf(-x);
                      const uint64_t ff = pair2(f, f);
                      WW.scale(pair2(f, f * f));
                      RS.scale(ff);
                      D1.scale(ff);
                      DV.scale(ff);
                      D2.scale(ff);
                      S += x;
                      x = 0.f;
                  }
                  const float w = expf(x);
                  const uint64_t ww = pair2(w, w);
                  const ulonglong2 kr = *reinterpret_cast<const ulonglong2*>(a + 4);     // (kio, rho) middle, low
                  const float4 v3 = *reinterpret_cast<const float4*>(a + 8);
                  uint64_t d = parts_diff(*reinterpret_cast<const uint64_t*>(a + 2), kr.x, kr.y, xh, xm, xl);
                  float dv = split2(parts_diff(pair2(v3.x, 0.f), pair2(v3.y, 0.f), pair2(v3.z, 0.f), pair2(xv.h, 0.f),
                                               pair2(xv.m, 0.f), pair2(xv.l, 0.f))).x;
                  if (v3.w != 0.f || x_out) {                  // a parameter that three floats do not hold
                      d = pair2(diff_f64(P.kio + entry, x0[0]), diff_f64(P.rho + entry, x0[1]));
                      dv = diff_f64(P.V + entry, x0[2]);
                  }
                  WW.add(ww, pair2(1.f, w));
                  RS.add(ww, pair2(resid, FREE ? s0 : 0.f));
                  const uint64_t wd = mul2(ww, d);             // rounded: it serves both sums
                  const float wdv = w * dv;
                  D1.add(wd, pair2(1.f, 1.f));
                  D2.add(wd, d);
                  DV.add(pair2(wdv, wdv), pair2(1.f, dv));
              };
              if (fits0) add(e0, o0 + Entry<N>::AUX, resid0, rw0, s00);
              if (fits1) add(e1, o1 + Entry<N>::AUX, resid1, rw1, s01);
          });
    if (!live) return;
    const int64_t n = P.n_vox;
    double* o = P.out;
    const double Wv = any ? WW.lo() : 0.0;
    const double Wd = fmax(Wv, 1e-300);
    const double s1[3] = {D1.lo(), D1.hi(), DV.lo()}, s2[3] = {D2.lo(), D2.hi(), DV.hi()};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const double a = s1[k] / Wd, b = s2[k] / Wd;
        o[(int64_t)k * n + v] = Wv > 0.0 ? x0[k] + a : 0.0;                      // kio, rho, V means
        o[(int64_t)(3 + k) * n + v] = Wv > 0.0 ? sqrt(fmax(b - a * a, 0.0)) : 0.0; // their std
    }
    o[6 * n + v] = Wv > 0.0 ? RS.lo() / Wd : 0.0;
    o[7 * n + v] = Wv > 0.0 ? Wv * Wv / fmax(WW.hi(), 1e-300) : 0.0;
    o[8 * n + v] = (FREE && Wv > 0.0) ? RS.hi() / Wd : 0.0;
}

template <int N, bool FREE, int THREADS, bool INDEXED>
static madi_status launch_kernel(const Plan& P, cudaStream_t s) {
    const auto kernel = bayes_kernel<N, FREE, THREADS, INDEXED>;
    constexpr int smem = CHUNK * Entry<N>::FLOATS * 4;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return host::cuda_fail(e, "bayes attribute");
    kernel<<<(unsigned)((P.n_vox + THREADS - 1) / THREADS), THREADS, smem, s>>>(P);
    e = cudaGetLastError();
    if (e != cudaSuccess) return host::cuda_fail(e, "bayes launch");
    return MADI_OK;
}

template <int N, bool FREE>
static madi_status launch(const madi_bayes_desc* d, const Plan& P, bool indexed, cudaStream_t s) {
    if (!indexed) return launch_kernel<N, FREE, 128, false>(P, s);
    const madi_status st = prune::build(P.ix, d->measured, d->lib, false, s);
    if (st != MADI_OK) return st;
    bayes_prep_kernel<N, FREE><<<(unsigned)((P.n_lib + 127) / 128), 128, 0, s>>>(P);
    // one warp a CTA until 128-thread CTAs give every SM four warps
    return P.n_vox < 152 * 128 ? launch_kernel<N, FREE, 32, true>(P, s) : launch_kernel<N, FREE, 128, true>(P, s);
}

template <bool FREE>
static madi_status launch_mode(const madi_bayes_desc* d, const Plan& P, bool indexed, cudaStream_t s) {
    switch ((d->n_feat + 3) / 4) {
        case 1: case 2: return launch<8, FREE>(d, P, indexed, s);
        case 3: case 4: return launch<16, FREE>(d, P, indexed, s);
        case 5: return launch<20, FREE>(d, P, indexed, s);
        case 6: return launch<24, FREE>(d, P, indexed, s);
        default: return launch<32, FREE>(d, P, indexed, s);
    }
}

static int entry_floats(int F) { return 2 * (F <= 8 ? 8 : F <= 16 ? 16 : F <= 20 ? 20 : F <= 24 ? 24 : 32) + 12; }

}  // namespace bayes
}  // namespace madi

using namespace madi;

void madi_match_column_mean(const float* lib, int32_t n_lib, int32_t n_feat, float* mu, cudaStream_t s);

// Fits that get room for the index.
static bool bayes_indexed(int64_t n_vox, int32_t n_lib) { return n_vox >= 64 && n_lib >= 256 && n_lib <= prune::MAX_LIB && n_vox < 0x7fffffff; }

// Where it pays for its ~0.06 ms: while the fit is one wave it saves a share of each
// voxel's entries (20 features, us without / with it: 500 voxels x 256 entries 100 /
// 145, x 600 206 / 220, x 1,000 331 / 305, x 5,000 1,575 / 1,134; 64 x 1,000 331 /
// 348, x 1,500 480 / 466), in larger ones also of the chip's work (50,000 x 256 145 /
// 149, x 400 216 / 181).  Five features and free S0 cross over at the same sizes, ten
// at 1,500 entries, with 15 % lost at 1,000.
static bool bayes_index_pays(int64_t n_vox, int32_t n_lib) { return n_lib >= (n_vox < 152 * 128 ? 1000 : 400); }

extern "C" int64_t madi_bayes_work_bytes(int64_t n_vox, int32_t n_lib, int32_t n_feat) {
    if (n_vox <= 0 || n_lib < 1 || n_feat < 1 || n_feat > 32 || !bayes_indexed(n_vox, n_lib)) return 256;
    prune::Index ix;
    return 256 + prune::layout(ix, nullptr, n_vox, n_lib, n_feat) + 4ll * n_lib * bayes::entry_floats(n_feat);
}

extern "C" int64_t madi_bayes_scratch_bytes(int32_t n_lib, int32_t n_feat) {
    (void)n_lib;
    (void)n_feat;
    return 256;                     // the column means
}

extern "C" madi_status madi_bayes(const madi_bayes_desc* d, void* stream) {
    host::clear_error();
    if (!d || !d->measured || !d->lib || !d->log_weight || !d->kio || !d->rho || !d->V || !d->out ||
        d->n_vox < 0 || d->n_lib < 1 || d->n_feat < 1)
        return host::fail(MADI_ERR_INVALID, "bayes: bad arguments");
    if (d->n_feat > 32) return host::fail(MADI_ERR_UNSUPPORTED, "bayes: at most 32 features");
    if (d->mode != MADI_MATCH_FIXED_S0 && d->mode != MADI_MATCH_FREE_S0)
        return host::fail(MADI_ERR_INVALID, "bayes: unknown mode");
    if (!(d->sigma_m > 0.0)) return host::fail(MADI_ERR_INVALID, "bayes: sigma_m must be > 0, got %g", d->sigma_m);
    const double inv = 1.0 / (2.0 * d->sigma_m * d->sigma_m);
    if (!(inv < 3.0e38)) return host::fail(MADI_ERR_UNSUPPORTED, "bayes: sigma_m %g too small for fp32 exponents", d->sigma_m);
    if (!d->scratch || d->scratch_bytes < 256) return host::fail(MADI_ERR_CAPACITY, "bayes: scratch < 256 bytes");
    if ((reinterpret_cast<uintptr_t>(d->scratch) & 255) != 0)
        return host::fail(MADI_ERR_INVALID, "bayes: scratch must be 256-byte aligned");
    if (d->n_vox == 0) return MADI_OK;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    float* mu = static_cast<float*>(d->scratch);
    if (d->mode == MADI_MATCH_FIXED_S0) {
        madi_match_column_mean(d->lib, d->n_lib, d->n_feat, mu, s);
    } else {
        const cudaError_t e = cudaMemsetAsync(mu, 0, 32 * sizeof(float), s);
        if (e != cudaSuccess) return host::cuda_fail(e, "bayes memset");
    }
    bayes::Plan P{};
    P.meas = d->measured;
    P.lib = d->lib;
    P.mu = mu;
    P.logq = d->log_weight;
    P.kio = d->kio;
    P.rho = d->rho;
    P.V = d->V;
    P.n_vox = d->n_vox;
    P.n_lib = d->n_lib;
    P.F = d->n_feat;
    P.inv2s2 = (float)inv;
    P.out = d->out;
    const bool indexed = bayes_indexed(d->n_vox, d->n_lib) && bayes_index_pays(d->n_vox, d->n_lib) &&
                         d->scratch_bytes >= madi_bayes_work_bytes(d->n_vox, d->n_lib, d->n_feat);
    if (indexed) {
        unsigned char* base = static_cast<unsigned char*>(d->scratch) + 256;
        const int64_t at = prune::layout(P.ix, base, d->n_vox, d->n_lib, d->n_feat);
        P.blocks = reinterpret_cast<float*>(base + at);
        P.ix.free_s0 = d->mode == MADI_MATCH_FREE_S0;
        P.ix.mu = P.ix.free_s0 ? nullptr : mu;
    }
    return d->mode == MADI_MATCH_FREE_S0 ? bayes::launch_mode<true>(d, P, indexed, s)
                                         : bayes::launch_mode<false>(d, P, indexed, s);
}
