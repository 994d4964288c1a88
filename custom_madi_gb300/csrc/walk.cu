// GB300 walker: one persistent launch walks every (ensemble, p_p) job of a
// batch.  Work unit = a tile of `tile_walkers` walkers (one per thread) of one
// job; CTAs pull tiles from a device counter and stage the tile's geometry
// (seeds, voxel candidate lists, cell facet table) into shared memory when it
// changes and fits.
//
// Per step and walker (fp32 state, madi/walker_gpu.py:574-655 transition):
//   propose x' = x + N(0, sigma^2 I)  (Philox4x32-10 + Box-Muller),
//   boundary: fatal escape (SI) or periodic wrap,
//   classify x' (the walker's label cache of three facet planes, else a
//   warp-cooperative pass over its cell's facets, else the voxel-grid rule,
//   else fp64),
//   m = endpoint membrane count, accept iff U64 < pp^m * 2^64, else revert,
//   Y'(t) = int_0^t (x - x0) dt by the step trapezoid (fp32 within one storage
//   interval, fp64 across intervals).
// At the end the phase epilogue forms dM = Y(delta) + Y(Delta) - Y(Delta+delta)
// per pair and axis and sums cos / sin(coef * u.dM) over the tile in exact
// 64-bit fixed point.
#include <cstdio>
#include <cstring>
#include <cmath>
#include "madi_device.cuh"
#include "madi_host.h"

namespace madi {

// Per Y grid point: coefficient k_p in {-1, 0, 1, 2} of Y(t_j) in the pair-p
// moment dM_p = Y(delta) + Y(Delta) - Y(Delta + delta), packed 2 bits per pair.
struct Snap { uint32_t code, any; };
MADI_DEV float snap_coef(uint32_t code, int p) { return (float)((int)((code >> (2 * p)) & 3u) - 1); }

// Y relative to x0 -> the reference's origin L/2 (madi/walker_gpu.py:562-564).
MADI_DEV double y_ref(double yrel, double x0, double half_L, double t) {
    return yrel + (x0 - half_L) * t;
}

// Shared-memory blocks of one CTA besides the staged geometry.
struct TileShared {
    long long* acc;       // [2 n_out] fixed-point cos / sin sums of the tile
    unsigned int* occ;    // [n_grid] inside counts
    const Snap* snap;     // [n_grid] moment coefficients
    double* auxd;         // [3][blockDim.x] Y' at the last storage point (fp64)
    float* auxf;          // [3 + 3 NP][blockDim.x] interval-start displacement, moments dM
    float4* fc;           // [6][blockDim.x] per-walker label cache (three facet planes + sphere)
    uint32_t* auxc;       // [2][blockDim.x] rare counters: accepted, rejected crossings
    float4* queue;        // [blockDim.x / 32][NGRP] walkers of the facet pass in flight
};

// Per-walker state touched once per storage interval lives in shared memory
// (structure of arrays, one column per thread) to keep the step loop in registers.
#define AUX_Y(k) ts.auxd[(k) * blockDim.x + threadIdx.x]
#define AUX_A(k) ts.auxf[(k) * blockDim.x + threadIdx.x]
#define AUX_M(p, k) ts.auxf[(3 + 3 * (p) + (k)) * blockDim.x + threadIdx.x]
#define AUX_C(k) ts.auxc[(k) * blockDim.x + threadIdx.x]
#define FC(k) ts.fc[(k) * blockDim.x + threadIdx.x]

// Per-walker label cache, built at a point q0 (w0 relative to the seed) by a full
// facet pass of cell c: facets k1, k2, k3 of smallest margin, every other facet's
// margin >= m4 as computed; T0 the error bound at q0, Tm = 3 T0.
//   FC(0..2) = facets k1, k2, k3 (n, h);   FC(3) = (w0, M = m4 - 5 T0);
//   FC(4) = (c, cell across k2);   FC(5) = (alpha_c - Tm, Tm, c, cell across k1).
// Another facet k has exact m_k(q0) >= m4 - T0 and is 1-Lipschitz, and the
// rounding of w and w0 moves |w - w0| by at most T(q) + T0, T(q) <= Tm while
// |w - w0| < L: so exact m_k(q) >= M - |w - w0|.  With mm, ms the smallest and
// second smallest cached margin at q (each within T(q)):
//   inside c     if mm > alpha_c + Tm and M - |w - w0| > alpha_c + Tm;
//   outside      if Tm <= mm < alpha_c - Tm and M - |w - w0| > Tm: q lies in the
//                Voronoi cell of c, short of its shrunk cell;
//   outside      if mm < Tm, mm > Tm - alpha_min, ms + mm > 2 Tm and M - |w - w0| >
//                max(-mm, 0) + Tm: q is within delta = max(-mm, 0) + Tm < alpha_min
//                of a point q' of the boundary of the cell of c (q moved back to
//                the one plane it is across, the other margins staying >= 0).  At
//                q' two seeds are nearest, so every seed i has a j with m_ij(q') <=
//                0, hence m_ij(q) <= delta < alpha_i: q is in no shrunk cell.
// (An extracellular walker's cell is never compared, so c serves for it.)
// A facet pass costs a warp ~1,900 cycles of latency and was 72 % of the walk (a
// free-water walk takes 73 ms where this one took 271: 64 entries x 25,000
// walkers), so the rules above go for fewer of them.  Misses: 12.3 % of
// walker-steps with the in / out rule of one sphere, 9.2 % with refused crossings
// settled on one plane, 7.0 % with the rule across a plane, 5.9 % with M kept
// instead of one radius (216 ms), 6.7 % with the first 16 slots deciding where
// they can, in half the loads and sorting (204 ms).
constexpr int FC_BYTES_PER_WALKER = 6 * 16;

// Sort key of a facet margin: the margin with the low KEY_BITS mantissa bits
// replaced by the facet's slot, compared as a float.  That moves the margin by
// at most 2^(KEY_BITS - 23) relative; key_floor() returns a lower bound of it.
constexpr int KEY_BITS = 6;                      // slots per cell <= 64
constexpr uint32_t KEY_SLOT = (1u << KEY_BITS) - 1u;

MADI_DEV float margin_key(float m, uint32_t slot) {
    return __uint_as_float((__float_as_uint(m) & ~KEY_SLOT) | slot);
}

MADI_DEV float key_floor(float key) {
    const uint32_t b = __float_as_uint(key);
    return __uint_as_float((b & 0x80000000u) ? (b | KEY_SLOT) : (b & ~KEY_SLOT));
}

MADI_DEV uint32_t key_slot(float key) { return __float_as_uint(key) & KEY_SLOT; }

MADI_DEV void cx(float& a, float& b) {
    const float lo = fminf(a, b), hi = fmaxf(a, b);
    a = lo; b = hi;
}

// ascending sort of four keys
MADI_DEV void sort4(float& a, float& b, float& c, float& d) {
    cx(a, b); cx(c, d); cx(a, c); cx(b, d); cx(b, c);
}

// the four smallest of two ascending quadruples, ascending, into (a0..a3)
MADI_DEV void merge4(float& a0, float& a1, float& a2, float& a3, float b0, float b1, float b2, float b3) {
    a0 = fminf(a0, b3); a1 = fminf(a1, b2); a2 = fminf(a2, b1); a3 = fminf(a3, b0);   // bitonic
    cx(a0, a2); cx(a1, a3); cx(a0, a1); cx(a2, a3);
}

// Full facet passes for the lanes with `need`, warp-cooperatively: a group of
// FG lanes takes one walker and FG FU of its cell's facet slots (FU coalesced
// loads per lane in flight), keeps each lane's four smallest margin keys with a
// sorting network and merges the group's in log2(FG) butterfly rounds.  The three
// smallest keys name the cached facets, whose margins are recomputed exactly (the
// true smallest margin is among them unless four margins lie within 2^-17 relative
// of each other, which the widened band covers); the fourth key bounds every other
// facet from below.  Slots are in order of h and m_k >= h_k - |w|, so the first 16
// slots decide whenever the last of them has h - |w| above the smallest margin
// (`rest`, which then bounds the slots not read); else the group reads the next
// 16 (each by its own need: caches and counts do not depend on the other walkers
// of the warp).  The group decides by the facet-plane rule and its first lane
// writes the walker's label cache.  A walker whose point lies across a facet is queued again from the
// cell beyond the most violated facet (at most three moves).  Called by all 32
// lanes; `start` is each walker's first cell; `refuse` marks walkers inside
// `start` whose acceptance number rejects any membrane crossing: a point outside
// that shrunk cell ends their pass as FACET_OUT of the same cell, whatever its own
// label.  Results: FACET_IN / FACET_OUT with cell_q set, or a negative code when
// the voxel-grid classifier has to decide.
// The pending walkers go to their groups through a queue in shared memory:
// (point, cell | lane << QLANE | refuse << QREFUSE).  Groups without a walker work
// on cell 0 and are ignored: a pass is one chain of ~1,000 cycles with no branch.
constexpr int FG = 4;
constexpr int FU = 4;
constexpr int NGRP = 32 / FG;
constexpr int VERDICT_MOVE = 8;
constexpr int QLANE = 24, QREFUSE = 29;          // a cell's slots take 640 B of a block < 4 GiB: cell < 2^23

template <bool PERIODIC>
MADI_DEV int coop_facets(const Geo& g, const TileShared& ts, bool need, float qx, float qy, float qz, int start,
                         bool refuse, int lane, int& cell_q) {
    const int gid = lane / FG, sub = lane % FG;
    const int warp0 = threadIdx.x & ~31;
    const int S = g.fstride;
    float4* queue = ts.queue + (threadIdx.x >> 5) * NGRP;
    int my_cell = start, hops = 0, r_mine = FACET_BAND;
    bool pend = need;
    unsigned pending = __ballot_sync(MADI_FULL, pend);
    while (pending) {
        const int rank = __popc(pending & ((1u << lane) - 1u));
        const bool mine = pend && rank < NGRP;
        if (mine) {
            const int tag = my_cell | (lane << QLANE) | ((refuse && hops == 0 ? 1 : 0) << QREFUSE);
            queue[rank] = make_float4(qx, qy, qz, __int_as_float(tag));
        }
        __syncwarp();
        const bool act = gid < __popc(pending);
        const float4 Q = queue[gid];
        const int tag = act ? __float_as_int(Q.w) : 0;
        const int sc = tag & ((1 << QLANE) - 1);
        const uint32_t base = (uint32_t)sc * (uint32_t)S;
        // the cell record and its first slots depend only on sc: one round trip
        const float4 cc = g.ccen[sc];
        float wx = 0.f, wy = 0.f, wz = 0.f, m1 = 0.f, T = 0.f, rest = 0.f;
        float q0 = 0.f, q1 = 0.f, q2 = 0.f, q3 = 0.f;
        float4 p1, p2, p3;
        int nb1 = -1, nb2 = -1, k0 = 0;
        bool more = true;                             // this group reads these slots (others: no key below infinity)
        do {
            float4 f[FU];
#pragma unroll
            for (int i = 0; i < FU; ++i) f[i] = g.fpl[base + k0 + sub + FG * i];
            if (k0 == 0) {
                wx = Q.x - cc.x; wy = Q.y - cc.y; wz = Q.z - cc.z;
                if (PERIODIC) {
                    const float hl = 0.5f * g.L;
                    wx = wx > hl ? wx - g.L : (wx < -hl ? wx + g.L : wx);
                    wy = wy > hl ? wy - g.L : (wy < -hl ? wy + g.L : wy);
                    wz = wz > hl ? wz - g.L : (wz < -hl ? wz + g.L : wz);
                }
            }
            float k[FU];
#pragma unroll
            for (int i = 0; i < FU; ++i)
                k[i] = more ? margin_key(facet_m(f[i], wx, wy, wz), (uint32_t)(k0 + sub + FG * i)) : __int_as_float(0x7f800000);
            sort4(k[0], k[1], k[2], k[3]);
#pragma unroll
            for (int o = 1; o < FG; o <<= 1) {
                const float b0 = __shfl_xor_sync(MADI_FULL, k[0], o);
                const float b1 = __shfl_xor_sync(MADI_FULL, k[1], o);
                const float b2 = __shfl_xor_sync(MADI_FULL, k[2], o);
                const float b3 = __shfl_xor_sync(MADI_FULL, k[3], o);
                merge4(k[0], k[1], k[2], k[3], b0, b1, b2, b3);
            }
            if (k0 == 0) { q0 = k[0]; q1 = k[1]; q2 = k[2]; q3 = k[3]; }
            else merge4(q0, q1, q2, q3, k[0], k[1], k[2], k[3]);
            const float h_last = __shfl_sync(MADI_FULL, f[FU - 1].w, lane | (FG - 1));
            // (a NaN margin's key names no slot of the cell)
            const uint32_t last = (uint32_t)S - 1u;
            const uint32_t k1 = base + min(key_slot(q0), last), k2 = base + min(key_slot(q1), last), k3 = base + min(key_slot(q2), last);
            // the three candidates' records and neighbours, loaded together (L1)
            p1 = g.fpl[k1]; p2 = g.fpl[k2]; p3 = g.fpl[k3];
            const int n1 = g.fnbr[k1], n2 = g.fnbr[k2], n3 = g.fnbr[k3];
            const float e1 = facet_m(p1, wx, wy, wz);
            const float e2 = facet_m(p2, wx, wy, wz);
            const float e3 = facet_m(p3, wx, wy, wz);
            m1 = fminf(e1, fminf(e2, e3));
            T = fmaf(2.0f * MADI_EPS21, fabsf(wx) + fabsf(wy) + fabsf(wz), g.ftol) + 7.62939453125e-6f * fabsf(m1);
            nb1 = e1 <= e2 ? (e1 <= e3 ? n1 : n3) : (e2 <= e3 ? n2 : n3);
            nb2 = n2;
            // |w| to 2^-22 relative, which T covers
            const float w2 = fmaf(wx, wx, fmaf(wy, wy, wz * wz));
            k0 += FG * FU;
            if (more)
                rest = k0 >= S ? 3.0e38f : (g.sorted ? h_last - w2 * rsqrtf(fmaxf(w2, 1e-30f)) - T : -3.0e38f);
            // the stride ends the loop: for a point that is not finite m1 + 2 T is NaN
            more = more && act && k0 < S && !(rest > m1 + 2.0f * T);
        } while (__any_sync(MADI_FULL, more));
        const float m4 = fminf(key_floor(q3), rest);
        const float dd = m1 - cc.w;
        int verdict = m1 > T ? (dd > T ? FACET_IN : (dd < -T ? FACET_OUT : FACET_BAND))
                             : (m1 < -T ? (nb1 >= 0 ? VERDICT_MOVE + nb1 : FACET_LEFT) : FACET_BAND);
        // nb1 < 0: an open cell's marker, no plane
        if (((tag >> QREFUSE) & 1) && dd < -T && nb1 >= 0) verdict = FACET_OUT;
        if (act && sub == 0 && (verdict == FACET_IN || verdict == FACET_OUT)) {
            const float Tm = 3.0f * T;
            const int n = blockDim.x;
            float4* fc = ts.fc + warp0 + ((tag >> QLANE) & 31);
            fc[0] = p1;
            fc[n] = p2;
            fc[2 * n] = p3;
            fc[3 * n] = make_float4(wx, wy, wz, fminf(m4 - 5.0f * T, g.L));
            fc[4 * n] = make_float4(cc.x, cc.y, cc.z, __int_as_float(nb2));
            fc[5 * n] = make_float4(cc.w - Tm, Tm, __int_as_float(sc), __int_as_float(nb1));
        }
        // each pending walker reads its group's verdict (group = its rank among the pending)
        const int v = __shfl_sync(MADI_FULL, verdict, (mine ? rank : 0) * FG);
        if (mine) {
            if (v >= VERDICT_MOVE && hops < 3) { my_cell = v - VERDICT_MOVE; ++hops; }
            else { r_mine = v >= VERDICT_MOVE ? FACET_LEFT : v; pend = false; }
        }
        __syncwarp();                                 // the queue is read before the next round writes it
        pending = __ballot_sync(MADI_FULL, pend);
    }
    cell_q = my_cell;
    return r_mine;
}

// Label of a point from the walker's cache (the rules above); true if they decide.
// `refuse`: the walker is inside `cell` and its acceptance number rejects any
// crossing, so a point outside that shrunk cell is as good as decided (reported
// as outside, whatever its own label): one plane with m < alpha_c - T(q) does,
// anywhere in the box (t_any >= T(q) while |w|_1 <= 3 L, which an infinite step
// does not pass).  Otherwise `start` becomes the cell beyond the cached
// facet k1 or k2 that the point lies farther across (exact planes of the cell).
template <bool PERIODIC>
MADI_DEV bool cached_label(const TileShared& ts, float L, float qx, float qy, float qz, bool refuse, int cell, float t_any,
                           float a_min, int& in, int& cell_q, int& start) {
    const float4 sp = FC(3), ce = FC(4), f1 = FC(0), f2 = FC(1), f3 = FC(2), th = FC(5);
    float wx = qx - ce.x, wy = qy - ce.y, wz = qz - ce.z;
    if (PERIODIC) {
        const float hl = 0.5f * L;
        wx = wx > hl ? wx - L : (wx < -hl ? wx + L : wx);
        wy = wy > hl ? wy - L : (wy < -hl ? wy + L : wy);
        wz = wz > hl ? wz - L : (wz < -hl ? wz + L : wz);
    }
    const float m1 = facet_m(f1, wx, wy, wz), m2 = facet_m(f2, wx, wy, wz), m3 = facet_m(f3, wx, wy, wz);
    const float mm = fminf(m1, fminf(m2, m3));
    const float ms = fmaxf(fminf(m1, m2), fminf(fmaxf(m1, m2), m3));
    const float ux = wx - sp.x, uy = wy - sp.y, uz = wz - sp.z;
    const float d2 = fmaf(ux, ux, fmaf(uy, uy, uz * uz));
    const float a_up = fmaf(2.0f, th.y, th.x);           // alpha_c + Tm
    const bool in_c = mm > a_up;
    const float r = sp.w - (in_c ? a_up : fmaxf(-mm, 0.f) + th.y);
    const bool near = r > 0.f && d2 < r * r * (1.0f - MADI_EPS19);
    const bool out = mm < th.x && (mm >= th.y || (mm > th.y - a_min && ms + mm > 2.0f * th.y));
    const int cc = __float_as_int(th.z);
    cell_q = cc;
    in = in_c ? 1 : 0;
    if (near && (in_c || out)) return true;
    if (refuse && cc == cell && mm < th.x - t_any && fabsf(wx) + fabsf(wy) + fabsf(wz) <= 3.0f * L) { in = 0; return true; }
    const int nb = __float_as_int(m1 <= m2 ? th.w : ce.w);
    if (!refuse && fminf(m1, m2) < -th.y && nb >= 0) start = nb;
    return false;
}

// Voxel-grid rule for the lanes with `need`, one warp-cooperative pass each, the
// fp64 rule where it cannot decide (a count in *fallbacks).  Rare (0.03 % of
// walker-steps), so a function of its own that rebuilds its view of the geometry:
// neither its registers nor the view's stay in the step loop.
struct FullLabel { int status, cell, inside; };

__device__ __noinline__ FullLabel full_labels(const madi_geometry* gd, const unsigned char* base, bool need, float qx,
                                              float qy, float qz, int guess, unsigned long long* fallbacks) {
    const int lane = threadIdx.x & 31;
    const Geo g = make_geo(*gd, base);
    int status = CLS_OK, seed = 0, inside = 0;
    for (unsigned pend = __ballot_sync(MADI_FULL, need); pend; pend &= pend - 1) {
        const int src = __ffs(pend) - 1;
        const float sx = __shfl_sync(MADI_FULL, qx, src);
        const float sy = __shfl_sync(MADI_FULL, qy, src);
        const float sz = __shfl_sync(MADI_FULL, qz, src);
        const int sg = __shfl_sync(MADI_FULL, guess, src);
        int s1 = 0, in = 0;
        int st = coop_classify(g, sx, sy, sz, sg, lane, s1, in);
        if (__any_sync(MADI_FULL, st == CLS_FALLBACK)) {
            st = coop_list_f64(g, sx, sy, sz, lane, s1, in);
            if (lane == 0) atomicAdd(fallbacks, 1ull);
        }
        if (lane == src) { status = st; seed = s1; inside = in; }
    }
    __syncwarp();
    return FullLabel{status, need && status == CLS_OK ? cell_of(g, seed) : 0, inside};
}

// Empties the walker's label cache.
MADI_DEV void clear_cache(const TileShared& ts) {
    FC(0) = FC(1) = FC(2) = make_float4(0.f, 0.f, 0.f, 3.0e38f);
    FC(3) = make_float4(0.f, 0.f, 0.f, -1.f);
    FC(4) = make_float4(0.f, 0.f, 0.f, __int_as_float(-1));
    FC(5) = make_float4(0.f, 0.f, __int_as_float(-1), __int_as_float(-1));
}

// The six normals of a step pair (the even step's first) and both acceptance words.
MADI_DEV void draw_pair(uint32_t widx, uint32_t pair, const madi_walk_job& job, float (&gv)[6], uint32_t& even, uint32_t& odd) {
    // the round keys are added up here: kept across steps they cost 20 registers
    uint32_t k0 = job.key0, k1 = job.key1;
    asm volatile("" : "+r"(k0), "+r"(k1));
    const U4 ra = philox10(U4{widx, pair, 0u, 0u}, k0, k1);
    const U4 rb = philox10(U4{widx, pair, 1u, 0u}, k0, k1);
    box_muller(ra.x, ra.y, gv[0], gv[1]);
    box_muller(ra.z, ra.w, gv[2], gv[3]);
    box_muller(rb.x, rb.y, gv[4], gv[5]);
    even = rb.z;
    odd = rb.w;
}

// Walk blockDim.x >> spread walkers of one job on geometry view g: 32 >> spread of
// them in the first lanes of each warp.  `local` is the lane's walker; lane groups
// beyond the first (SPREAD) hold the same walkers' numbers and no walker.
template <int OUT, bool PERIODIC, int NP, bool SPREAD>
__device__ __forceinline__ void walk_tile(const madi_walk_desc& d, const madi_walk_job& job,
                                          const madi_geometry& gd, const unsigned char* base, int local, int spread,
                                          const TileShared& ts) {
    const int lane = threadIdx.x & 31;
    const Geo g = make_geo(gd, base);
    const bool active = local < job.n_walkers && (!SPREAD || lane < (32 >> spread));
    const uint32_t widx = job.walker_base + (uint32_t)local;
    // fp64 is ~2 lanes a cycle: conversions and compares of the descriptor's doubles
    // are done here once (the empty asm keeps them from being redone in each step,
    // where they held 31 % of the fp64 pipe: 204 -> 199 ms, 64 entries x 25,000
    // walkers; 4.98 -> 4.71 ms, one entry x 10,000)
    float L = (float)gd.L, sigma = (float)d.sigma;
    asm volatile("" : "+f"(L), "+f"(sigma));
    const bool cells = gd.has_cells != 0;
    const bool stream = d.rng == MADI_RNG_STREAM;

    // ---- initial position (Omega_src cube; the whole box when periodic) ----
    float px = 0.f, py = 0.f, pz = 0.f;
    if (active) {
        double x0, y0, z0;
        if (stream) {
            x0 = d.init[3 * (size_t)local + 0];
            y0 = d.init[3 * (size_t)local + 1];
            z0 = d.init[3 * (size_t)local + 2];
        } else {
            const U4 r = philox10(U4{widx, 0u, 0u, 1u}, job.key0, job.key1);
            const double span = gd.source_hi - gd.source_lo;
            x0 = gd.source_lo + span * ((double)r.x * 2.3283064365386963e-10);
            y0 = gd.source_lo + span * ((double)r.y * 2.3283064365386963e-10);
            z0 = gd.source_lo + span * ((double)r.z * 2.3283064365386963e-10);
        }
        px = (float)x0; py = (float)y0; pz = (float)z0;
        if (PERIODIC) {
            if (px >= L) px = 0.f;
            if (py >= L) py = 0.f;
            if (pz >= L) pz = 0.f;
        }
    }
    const float x0f = px, y0f = py, z0f = pz;
    // ---- state ----
    float dx = 0.f, dy = 0.f, dz = 0.f;           // unwrapped displacement from x0
    int cell = 0, inside = 0;                     // Voronoi cell of the position and its label
    const bool facets = cells && g.n_cells > 0;
    bool dead = !active;
    bool frozen = !active;
    uint32_t n_full = 0, n_t1 = 0, n_fp = 0, escaped = 0, cerr = 0;
#pragma unroll
    for (int k = 0; k < 3; ++k) { AUX_Y(k) = 0.0; AUX_A(k) = 0.f; }
    AUX_C(0) = AUX_C(1) = 0u;
    unsigned long long* const cnt = reinterpret_cast<unsigned long long*>(d.counters + (size_t)job.slot * MADI_CNT_N);
#pragma unroll
    for (int p = 0; p < NP; ++p) { AUX_M(p, 0) = 0.f; AUX_M(p, 1) = 0.f; AUX_M(p, 2) = 0.f; }
    clear_cache(ts);
    if (cells) {
        const FullLabel f = full_labels(&gd, base, active, px, py, pz, -1, &cnt[MADI_CNT_FALLBACK64]);
        if (active) {
            if (f.status != CLS_OK) { cerr = 1; dead = true; }
            else { cell = f.cell; inside = f.inside; }
            ++n_full;
        }
    }
    float Sx = 0.f, Sy = 0.f, Sz = 0.f;           // sum of displacements in this interval
    const size_t row = (size_t)job.y_row + (size_t)local;
    if (OUT == MADI_OUT_Y && active) {
        d.Y[(row * d.n_grid) * 3 + 0] = 0.0;
        d.Y[(row * d.n_grid) * 3 + 1] = 0.0;
        d.Y[(row * d.n_grid) * 3 + 2] = 0.0;
        d.inside_trace[row * d.n_grid] = (int8_t)inside;
    }
    {
        const unsigned b = __ballot_sync(0xffffffffu, active && inside);
        if (lane == 0 && b) atomicAdd(&ts.occ[0], (unsigned)__popc(b));
    }
    int always = job.pp >= 1.0;
    asm volatile("" : "+r"(always));
    const uint32_t th1 = (uint32_t)(job.thr1 >> 32), th2 = (uint32_t)(job.thr2 >> 32);
    // error bound of any facet margin in the box (|w|_1 <= 3 L)
    float t_any = fmaf(6.0f * MADI_EPS21, L, (float)gd.facet_tol);
    asm volatile("" : "+f"(t_any));
    const float a_min = alpha_bound(gd);
    float gv[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    uint32_t acc_word = 0, acc_word_odd = 0;
    int h_left = d.steps_per_h;
    int jgrid = 0;
#pragma unroll 1
    for (int step = 0; step < d.n_steps; ++step) {
        // ---- random numbers: one Philox call per step on average ----
        float nx, ny, nz;
        uint32_t word = 0;
        bool u_ge1 = false, u_lt1 = false, u_lt2 = false;
        if (stream) {
            if (!dead) {
                const size_t o = ((size_t)step * job.n_walkers + local);
                nx = (float)d.incr[3 * o + 0];
                ny = (float)d.incr[3 * o + 1];
                nz = (float)d.incr[3 * o + 2];
                const double u = d.unif[o];
                u_ge1 = u >= job.pp; u_lt1 = u < job.pp; u_lt2 = u < job.pp * job.pp;
            } else { nx = ny = nz = 0.f; }
        } else if (SPREAD) {
            // lane group i draws step pair i of 1 << spread pairs; each step reads its pair's
            if ((step & ((2 << spread) - 1)) == 0)
                draw_pair(widx, ((uint32_t)step >> 1) + ((uint32_t)lane >> (5 - spread)), job, gv, acc_word, acc_word_odd);
            const int from = (lane & (31 >> spread)) | (((step >> 1) & ((1 << spread) - 1)) << (5 - spread));
            const bool odd = step & 1;
            nx = __shfl_sync(MADI_FULL, odd ? gv[3] : gv[0], from) * sigma;
            ny = __shfl_sync(MADI_FULL, odd ? gv[4] : gv[1], from) * sigma;
            nz = __shfl_sync(MADI_FULL, odd ? gv[5] : gv[2], from) * sigma;
            word = __shfl_sync(MADI_FULL, odd ? acc_word_odd : acc_word, from);
        } else if ((step & 1) == 0) {
            draw_pair(widx, (uint32_t)step >> 1, job, gv, word, acc_word_odd);
            nx = gv[0] * sigma; ny = gv[1] * sigma; nz = gv[2] * sigma;
        } else {
            nx = gv[3] * sigma; ny = gv[4] * sigma; nz = gv[5] * sigma;
            word = acc_word_odd;
        }
        // ---- proposal and boundary ----
        float qx = px, qy = py, qz = pz;
        bool ok = false;
        if (!dead) {
            qx = px + nx; qy = py + ny; qz = pz + nz;
            ok = true;
            if (PERIODIC) {
                if (qx < 0.f) qx += L;
                if (qx >= L) qx -= L;
                if (qy < 0.f) qy += L;
                if (qy >= L) qy -= L;
                if (qz < 0.f) qz += L;
                if (qz >= L) qz -= L;
            } else if (qx < 0.f || qx >= L || qy < 0.f || qy >= L || qz < 0.f || qz >= L) {
                ok = false;
                escaped = 1;
                dead = true;
            }
        }
        const float ex = dx + nx, ey = dy + ny, ez = dz + nz;
        // ---- label from the cached facet planes ----
        const bool refuse = inside && !always && (stream ? u_ge1 : word > th1);
        bool t1 = false;
        int t1_in = 0, t1_cell = cell;
        int start = cell;
        if (ok && facets)
            t1 = cached_label<PERIODIC>(ts, L, qx, qy, qz, refuse, cell, t_any, a_min, t1_in, t1_cell, start);
        // ---- cache misses: cooperative full facet passes, which rebuild the caches ----
        const bool miss = ok && facets && !t1;
        n_fp += miss ? 1u : 0u;
        if (__any_sync(MADI_FULL, miss)) {
            int cq = start;
            const int r = coop_facets<PERIODIC>(g, ts, miss, qx, qy, qz, start, refuse, lane, cq);
            if (miss && r >= 0) { t1 = true; t1_in = r; t1_cell = cq; }
        }
        // ---- full classifications of this step ----
        const bool need = ok && cells && !t1;
        FullLabel full{CLS_OK, 0, 0};
        if (__any_sync(MADI_FULL, need)) full = full_labels(&gd, base, need, qx, qy, qz, cell, &cnt[MADI_CNT_FALLBACK64]);
        if (ok) {
            int ncell = 0, nin = 0;
            if (t1) {
                ncell = t1_cell; nin = t1_in; ++n_t1;
            } else if (need) {
                ++n_full;
                if (full.status != CLS_OK) { cerr = 1; dead = true; }
                else { ncell = full.cell; nin = full.inside; }
            }
            if (!dead) {
                int m = 0;
                if (inside != nin) m = 1;
                else if (inside && nin && cell != ncell) m = 2;
                bool accept = true;
                if (m > 0 && !always) {
                    if (stream) {
                        accept = m == 1 ? u_lt1 : u_lt2;
                    } else {
                        const uint32_t th = m == 1 ? th1 : th2;
                        if (word != th) {
                            accept = word < th;
                        } else {
                            const uint64_t thr = m == 1 ? job.thr1 : job.thr2;
                            const U4 rc = philox10(U4{widx, (uint32_t)step, 2u, 0u}, job.key0, job.key1);
                            accept = rc.x < (uint32_t)thr;
                        }
                    }
                    ++AUX_C(accept ? 0 : 1);
                }
                if (accept) {
                    px = qx; py = qy; pz = qz;
                    dx = ex; dy = ey; dz = ez;
                    cell = ncell; inside = nin;
                }
            }
        }
        if (!dead) {
            Sx += dx; Sy += dy; Sz += dz;
        } else if (!frozen) {
            // Walker stopped (fatal escape or classifier failure): close its
            // trapezoid at the last accepted step and add nothing after.
            frozen = true;
            AUX_Y(0) += d.ts * ((double)Sx + 0.5 * ((double)AUX_A(0) - (double)dx));
            AUX_Y(1) += d.ts * ((double)Sy + 0.5 * ((double)AUX_A(1) - (double)dy));
            AUX_Y(2) += d.ts * ((double)Sz + 0.5 * ((double)AUX_A(2) - (double)dz));
            Sx = Sy = Sz = 0.f;
            AUX_A(0) = dx; AUX_A(1) = dy; AUX_A(2) = dz;
        }
        if (--h_left == 0) {
            h_left = d.steps_per_h;
            ++jgrid;
            const double tsd = d.ts;
            const double Yx = AUX_Y(0) + tsd * ((double)Sx + 0.5 * ((double)AUX_A(0) - (double)dx));
            const double Yy = AUX_Y(1) + tsd * ((double)Sy + 0.5 * ((double)AUX_A(1) - (double)dy));
            const double Yz = AUX_Y(2) + tsd * ((double)Sz + 0.5 * ((double)AUX_A(2) - (double)dz));
            AUX_Y(0) = Yx; AUX_Y(1) = Yy; AUX_Y(2) = Yz;
            Sx = Sy = Sz = 0.f;
            AUX_A(0) = dx; AUX_A(1) = dy; AUX_A(2) = dz;
            if (OUT == MADI_OUT_Y) {
                if (active) {
                    const double t = (double)jgrid * d.steps_per_h * tsd;
                    const double half_L = 0.5 * gd.L;
                    double* yo = d.Y + (row * d.n_grid + jgrid) * 3;
                    yo[0] = y_ref(Yx, x0f, half_L, t);
                    yo[1] = y_ref(Yy, y0f, half_L, t);
                    yo[2] = y_ref(Yz, z0f, half_L, t);
                    d.inside_trace[row * d.n_grid + jgrid] = (int8_t)inside;
                }
            } else {
                const Snap sn = ts.snap[jgrid];
                if (sn.any) {
                    const float fx = (float)Yx, fy = (float)Yy, fz = (float)Yz;
#pragma unroll
                    for (int p = 0; p < NP; ++p) {
                        const float k = snap_coef(sn.code, p);
                        if (k != 0.f) {
                            AUX_M(p, 0) = fmaf(k, fx, AUX_M(p, 0));
                            AUX_M(p, 1) = fmaf(k, fy, AUX_M(p, 1));
                            AUX_M(p, 2) = fmaf(k, fz, AUX_M(p, 2));
                        }
                    }
                }
            }
            const unsigned b = __ballot_sync(0xffffffffu, active && inside);
            if (lane == 0 && b) atomicAdd(&ts.occ[jgrid], (unsigned)__popc(b));
        }
    }
    // ---- phase epilogue: per (pair, dir, b) warp sums -> fixed point ----
    if (OUT == MADI_OUT_FUSED) {
        bool live = active && !escaped && !cerr;
        int from = threadIdx.x;
        bool mine = true;
        if (SPREAD) {
            // the sums are those of the launch without lane groups: 32 walkers to a warp again
            FC(0).x = live ? 1.f : 0.f;
            __syncthreads();
            const int per = 5 - spread;
            mine = from < (int)(blockDim.x >> spread);
            from = ((from >> per) << 5) | (from & ((1 << per) - 1));
            if (mine) live = ts.fc[from].x != 0.f;
        }
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            if (p >= d.n_pairs || !mine) break;
            const float* m = &ts.auxf[(3 + 3 * p) * blockDim.x + from];
            const float mx = m[0], my = m[blockDim.x], mz = m[2 * blockDim.x];
            for (int u = 0; u < d.n_dirs; ++u) {
                const float proj = fmaf(d.dirs[3 * u], mx, fmaf(d.dirs[3 * u + 1], my, d.dirs[3 * u + 2] * mz));
                for (int bb = 0; bb < d.n_b; ++bb) {
                    float c = 0.f, s = 0.f;
                    if (live) sincosf(d.coef[p * d.n_b + bb] * proj, &s, &c);
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) {
                        c += __shfl_xor_sync(0xffffffffu, c, o);
                        s += __shfl_xor_sync(0xffffffffu, s, o);
                    }
                    if (lane == 0) {
                        const int idx = ((p * d.n_b + bb) * d.n_dirs + u) * 2;
                        atomicAdd(reinterpret_cast<unsigned long long*>(&ts.acc[idx]),
                                  (unsigned long long)__float2ll_rn(c * 4294967296.0f));
                        atomicAdd(reinterpret_cast<unsigned long long*>(&ts.acc[idx + 1]),
                                  (unsigned long long)__float2ll_rn(s * 4294967296.0f));
                    }
                }
            }
        }
    }
    // ---- counters ----
    {
        const uint32_t v0 = __reduce_add_sync(0xffffffffu, active ? 1u : 0u);
        const uint32_t v1 = __reduce_add_sync(0xffffffffu, escaped);
        const uint32_t v2 = __reduce_add_sync(0xffffffffu, cerr);
        const uint32_t v3 = __reduce_add_sync(0xffffffffu, n_full);
        const uint32_t v4 = __reduce_add_sync(0xffffffffu, n_t1);
        const uint32_t v6 = __reduce_add_sync(0xffffffffu, AUX_C(0));
        const uint32_t v7 = __reduce_add_sync(0xffffffffu, AUX_C(1));
        const uint32_t v8 = __reduce_add_sync(0xffffffffu, n_fp);
        if (lane == 0) {
            if (v0) atomicAdd(&cnt[MADI_CNT_WALKERS], (unsigned long long)v0);
            if (v1) atomicAdd(&cnt[MADI_CNT_ESCAPED], (unsigned long long)v1);
            if (v2) atomicAdd(&cnt[MADI_CNT_CLASSIFIER_ERROR], (unsigned long long)v2);
            if (v3) atomicAdd(&cnt[MADI_CNT_FULL], (unsigned long long)v3);
            if (v4) atomicAdd(&cnt[MADI_CNT_TIER1], (unsigned long long)v4);
            if (v6) atomicAdd(&cnt[MADI_CNT_CROSS_ACCEPT], (unsigned long long)v6);
            if (v7) atomicAdd(&cnt[MADI_CNT_CROSS_REJECT], (unsigned long long)v7);
            if (v8) atomicAdd(&cnt[MADI_CNT_FACET_PASS], (unsigned long long)v8);
        }
    }
}

constexpr int SPREAD_THREADS = 128;

template <int OUT, bool PERIODIC, int NP, int MINB, bool SPREAD>
__global__ void __launch_bounds__(SPREAD ? SPREAD_THREADS : 256, MINB) walk_f32_kernel(const __grid_constant__ madi_walk_desc d, int spread) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_item;
    const int nthr = blockDim.x;
    const int tid = threadIdx.x;
    const int n_out = d.n_pairs * d.n_b * d.n_dirs;
    if (!SPREAD) spread = 0;
    const int parts = SPREAD ? (d.tile_walkers << spread) / SPREAD_THREADS : 1;      // CTAs' shares of a tile
    const int n_items = d.n_tiles * parts;
    // Dynamic shared memory: [stage][acc int64 x 2 n_out][occ u32 x n_grid][snap x n_grid]
    unsigned char* stage = smem;
    TileShared ts;
    ts.acc = reinterpret_cast<long long*>(smem + d.stage_smem);
    ts.occ = reinterpret_cast<unsigned int*>(ts.acc + 2 * n_out);
    Snap* snap = reinterpret_cast<Snap*>(ts.occ + d.n_grid);
    ts.snap = snap;
    unsigned char* aux = smem + d.stage_smem + 16 * n_out + 12 * ((d.n_grid + 3) & ~3);
    ts.auxd = reinterpret_cast<double*>(aux);
    ts.fc = reinterpret_cast<float4*>(aux + 24 * nthr);
    ts.auxf = reinterpret_cast<float*>(aux + (24 + FC_BYTES_PER_WALKER) * nthr);
    ts.auxc = reinterpret_cast<uint32_t*>(ts.auxf + (3 + 3 * NP) * nthr);
    ts.queue = reinterpret_cast<float4*>(ts.auxc + 2 * nthr);    // the 4 bytes a walker left of the 12

    for (int j = tid; j < d.n_grid; j += nthr) {
        uint32_t code = 0, any = 0;
        for (int p = 0; p < MADI_MAX_PAIRS; ++p) {
            int k = 0;
            if (p < d.n_pairs) k = (d.pair_jd[p] == j) + (d.pair_jD[p] == j) - (d.pair_js[p] == j);
            code |= (uint32_t)(k + 1) << (2 * p);
            any |= k != 0;
        }
        snap[j] = Snap{code, any};
    }
    int cur_geom = -1;
    int first = 1;
    for (;;) {
        __syncthreads();
        if (tid == 0) {
            if (d.grid_blocks > 0) s_item = (int)atomicAdd(d.work_counter, 1u);
            else s_item = first ? (int)blockIdx.x : n_items;
        }
        first = 0;
        for (int i = tid; i < 2 * n_out; i += nthr) ts.acc[i] = 0;
        for (int j = tid; j < d.n_grid; j += nthr) ts.occ[j] = 0;
        __syncthreads();
        const int item = s_item;
        if (item >= n_items) break;
        const int tile = item / parts;
        const int jn = find_job(d.jobs, d.n_jobs, tile);
        const madi_walk_job job = d.jobs[jn];
        const madi_geometry gd = d.geoms[job.geom];
        const int local = SPREAD ? (((item - job.tile_begin * parts) * nthr + (tid & ~31)) >> spread) + (tid & (31 >> spread))
                                 : (tile - job.tile_begin) * nthr + tid;
        const bool here = d.stage_smem > 0 && (int)gd.stage_bytes <= d.stage_smem;
        if (here && job.geom != cur_geom) {
            const uint4* src = reinterpret_cast<const uint4*>(gd.stage);
            uint4* dst = reinterpret_cast<uint4*>(stage);
            for (uint32_t i = tid; i < gd.stage_bytes / 16u; i += nthr) dst[i] = src[i];
            cur_geom = job.geom;
        }
        __syncthreads();
        walk_tile<OUT, PERIODIC, NP, SPREAD>(d, job, d.geoms[job.geom],
                                             here ? stage : reinterpret_cast<const unsigned char*>(gd.stage), local, spread, ts);
        __syncthreads();
        if (OUT == MADI_OUT_FUSED) {
            long long* out = reinterpret_cast<long long*>(d.accum) + (size_t)job.slot * 2 * n_out;
            for (int i = tid; i < 2 * n_out; i += nthr)
                if (ts.acc[i]) atomicAdd(reinterpret_cast<unsigned long long*>(&out[i]), (unsigned long long)ts.acc[i]);
        }
        uint64_t* occ_out = d.occupancy + (size_t)job.slot * d.n_grid;
        for (int j = tid; j < d.n_grid; j += nthr)
            if (ts.occ[j]) atomicAdd(reinterpret_cast<unsigned long long*>(&occ_out[j]), (unsigned long long)ts.occ[j]);
    }
}

// ---------------------------------------------------------------------------
// fp64 walker (madi/walker_gpu.py:520-585 design and :698-840 arithmetic:
// separately rounded fp64, reference origin L/2, Y stored).  One thread per
// walker of jobs[0]; it replays a fixed random stream (golden check) or walks
// the fp32 walker's Philox numbers.
//
// Labels are the exact KD rule's at every step.  The rule itself (a stackless
// fp64 descent, a chain of dependent loads and fp64 operations per node) took
// 97 % of the walk, so the label comes from the fp32 walker's facet planes where
// their margins clear the error band (its allowance of 2^-21 L covers rounding
// the fp64 point to fp32, sqrt(3) 2^-24 L), and from the KD rule in the rest
// (~0.04 % of steps).  What remains is bound by the fp64 pipe: Box-Muller in
// fp64, once per pair of steps.  16,000 walkers x 4,600 steps in a 64-cell box:
// ~900 ms before, 33 ms now.
// ---------------------------------------------------------------------------
constexpr int F64_THREADS = 128;

// The six normals of step pair `pair` of walker widx from the Philox stream of
// the fp32 walker, in fp64 (Box-Muller: u1 = (w + 1/2) 2^-32, u2 = (w' >> 8)
// 2^-24; the first three are the even step's), and the two acceptance words: the
// fp32 walker's random numbers, evaluated in the reference's precision.
MADI_DEV void normals_f64(uint32_t widx, uint32_t pair, uint32_t k0, uint32_t k1, double (&gv)[6], uint32_t (&word)[2]) {
    const U4 ra = philox10(U4{widx, pair, 0u, 0u}, k0, k1);
    const U4 rb = philox10(U4{widx, pair, 1u, 0u}, k0, k1);
    const uint32_t wd[6] = {ra.x, ra.y, ra.z, ra.w, rb.x, rb.y};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const double u1 = __dadd_rn(__dmul_rn((double)wd[2 * k], 2.3283064365386963e-10), 1.1641532182693481e-10);
        const double u2 = __dmul_rn((double)(wd[2 * k + 1] >> 8), 5.9604644775390625e-08);
        const double r = sqrt(__dmul_rn(-2.0, log(u1)));
        double sn, cs;
        sincos(__dmul_rn(6.283185307179586, u2), &sn, &cs);
        gv[2 * k] = __dmul_rn(r, cs);
        gv[2 * k + 1] = __dmul_rn(r, sn);
    }
    word[0] = rb.z;
    word[1] = rb.w;
}

__global__ void __launch_bounds__(F64_THREADS) walk_f64_kernel(const madi_walk_desc d) {
    __shared__ float4 s_fc[FC_BYTES_PER_WALKER / 16 * F64_THREADS], s_queue[F64_THREADS / 32 * NGRP];
    TileShared ts{};
    ts.fc = s_fc;
    ts.queue = s_queue;
    const madi_walk_job job = d.jobs[0];
    const int lane = threadIdx.x & 31;
    const int w0 = blockIdx.x * blockDim.x + threadIdx.x;
    if (w0 - lane >= job.n_walkers) return;                  // whole warps only: the facet pass is warp-wide
    const bool active = w0 < job.n_walkers;
    const int w = active ? w0 : job.n_walkers - 1;           // spare lanes shadow the last walker, write nothing
    const madi_geometry gd = d.geoms[job.geom];
    const Geo g = make_geo(gd, reinterpret_cast<const unsigned char*>(gd.stage));
    const bool periodic = gd.boundary == MADI_BOUNDARY_PERIODIC;
    const bool cells = gd.has_cells != 0;
    const bool stream = d.rng == MADI_RNG_STREAM;
    const uint32_t widx = job.walker_base + (uint32_t)w;
    const double L = gd.L, half_L = gd.L / 2.0, ts_ms = d.ts, pp = job.pp;
    const size_t row = (size_t)job.y_row + w;
    double px, py, pz;
    if (stream) {
        px = d.init[3 * (size_t)w]; py = d.init[3 * (size_t)w + 1]; pz = d.init[3 * (size_t)w + 2];
    } else {
        const U4 r = philox10(U4{widx, 0u, 0u, 1u}, job.key0, job.key1);
        const double span = gd.source_hi - gd.source_lo;
        px = gd.source_lo + span * ((double)r.x * 2.3283064365386963e-10);
        py = gd.source_lo + span * ((double)r.y * 2.3283064365386963e-10);
        pz = gd.source_lo + span * ((double)r.z * 2.3283064365386963e-10);
        if (periodic) {
            if (px >= L) px = 0.0;
            if (py >= L) py = 0.0;
            if (pz >= L) pz = 0.0;
        }
    }
    const bool facets = cells && gd.n_cells > 0;
    const float Lf = (float)L, a_min = alpha_bound(gd);
    clear_cache(ts);
    int cell = 0, inside = 0, escaped = 0, cerr = 0;
    uint32_t n_acc = 0, n_rej = 0, n_full = 0;
    if (cells) {
        int s1 = 0;
        if (classify_kd_f64(g, px, py, pz, s1, inside) != CLS_OK) cerr = 1;
        cell = g.cell[s1];
        ++n_full;
    }
    int kx = 0, ky = 0, kz = 0;
    double xp = __dsub_rn(px, half_L), yp = __dsub_rn(py, half_L), zp = __dsub_rn(pz, half_L);
    double Yx = 0.0, Yy = 0.0, Yz = 0.0;
    double* Yo = d.Y + row * d.n_grid * 3;
    int8_t* It = d.inside_trace + row * d.n_grid;
    if (active) {
        Yo[0] = Yo[1] = Yo[2] = 0.0;
        It[0] = (int8_t)inside;
    }
    double gv[6];
    uint32_t words[2] = {0u, 0u};
    for (int step = 0; step < d.n_steps; ++step) {
        const bool alive = active && !escaped && !cerr;
        double qx = px, qy = py, qz = pz, u = 0.0;
        int qkx = kx, qky = ky, qkz = kz;
        uint32_t word = 0;
        bool ok = alive;
        if (alive) {
            double inc[3];
            if (stream) {
                const size_t o = (size_t)step * job.n_walkers + w;
                inc[0] = d.incr[3 * o]; inc[1] = d.incr[3 * o + 1]; inc[2] = d.incr[3 * o + 2];
                u = d.unif[o];
            } else {
                if ((step & 1) == 0) {
                    normals_f64(widx, (uint32_t)step >> 1, job.key0, job.key1, gv, words);
                } else {
#pragma unroll
                    for (int i = 0; i < 3; ++i) gv[i] = gv[3 + i];
                }
                word = words[step & 1];
                inc[0] = __dmul_rn(gv[0], d.sigma); inc[1] = __dmul_rn(gv[1], d.sigma); inc[2] = __dmul_rn(gv[2], d.sigma);
            }
            qx = __dadd_rn(px, inc[0]); qy = __dadd_rn(py, inc[1]); qz = __dadd_rn(pz, inc[2]);
            if (periodic) {
                if (qx < 0.0) { qx = __dadd_rn(qx, L); --qkx; }
                if (qx >= L) { qx = __dsub_rn(qx, L); ++qkx; }
                if (qy < 0.0) { qy = __dadd_rn(qy, L); --qky; }
                if (qy >= L) { qy = __dsub_rn(qy, L); ++qky; }
                if (qz < 0.0) { qz = __dadd_rn(qz, L); --qkz; }
                if (qz >= L) { qz = __dsub_rn(qz, L); ++qkz; }
            } else if (qx < 0.0 || qx >= L || qy < 0.0 || qy >= L || qz < 0.0 || qz >= L) {
                escaped = 1;
                ok = false;
            }
        }
        // ---- label: facet planes (cache, then a warp-wide pass), else the KD rule ----
        int ncell = 0, nin = 0;
        bool known = !cells;
        if (facets) {
            const float fx = (float)qx, fy = (float)qy, fz = (float)qz;
            // a step longer than the box leaves a periodic point outside after one wrap
            const bool boxed = ok && fx >= 0.f && fx <= Lf && fy >= 0.f && fy <= Lf && fz >= 0.f && fz <= Lf;     // no NaN
            int start = cell;
            // (no early refusal here: `refuse` is false)
            if (boxed) known = periodic ? cached_label<true>(ts, Lf, fx, fy, fz, false, cell, 0.f, a_min, nin, ncell, start)
                                        : cached_label<false>(ts, Lf, fx, fy, fz, false, cell, 0.f, a_min, nin, ncell, start);
            const bool miss = boxed && !known;
            if (__any_sync(MADI_FULL, miss)) {
                int cq = start;
                const int r = periodic ? coop_facets<true>(g, ts, miss, fx, fy, fz, start, false, lane, cq)
                                       : coop_facets<false>(g, ts, miss, fx, fy, fz, start, false, lane, cq);
                if (miss && r >= 0) { known = true; nin = r; ncell = cq; }
            }
        }
        if (ok) {
            if (!known) {
                int s1 = 0;
                if (classify_kd_f64(g, qx, qy, qz, s1, nin) != CLS_OK) { cerr = 1; }
                ncell = g.cell[s1];
            }
            if (cells) ++n_full;
            if (!cerr) {
                int m = 0;
                if (inside && !nin) m = 1;
                else if (!inside && nin) m = 1;
                else if (inside && nin && cell != ncell) m = 2;
                bool accept = true;
                if (m > 0 && pp < 1.0) {
                    if (stream) {
                        const double thr = m == 1 ? pp : __dmul_rn(pp, pp);
                        accept = !(u >= thr);
                    } else {            // 64-bit uniform against floor(pp^m 2^64), as the fp32 walker
                        const uint64_t thr = m == 1 ? job.thr1 : job.thr2;
                        const uint32_t th = (uint32_t)(thr >> 32);
                        if (word != th) {
                            accept = word < th;
                        } else {
                            const U4 rc = philox10(U4{widx, (uint32_t)step, 2u, 0u}, job.key0, job.key1);
                            accept = rc.x < (uint32_t)thr;
                        }
                    }
                    if (accept) ++n_acc; else ++n_rej;
                }
                if (accept) {
                    px = qx; py = qy; pz = qz; kx = qkx; ky = qky; kz = qkz;
                    cell = ncell; inside = nin;
                }
                double xn = __dsub_rn(px, half_L), yn = __dsub_rn(py, half_L), zn = __dsub_rn(pz, half_L);
                if (periodic) {
                    xn = __dadd_rn(xn, __dmul_rn((double)kx, L));
                    yn = __dadd_rn(yn, __dmul_rn((double)ky, L));
                    zn = __dadd_rn(zn, __dmul_rn((double)kz, L));
                }
                Yx = __dadd_rn(Yx, __dmul_rn(__dmul_rn(0.5, __dadd_rn(xp, xn)), ts_ms));
                Yy = __dadd_rn(Yy, __dmul_rn(__dmul_rn(0.5, __dadd_rn(yp, yn)), ts_ms));
                Yz = __dadd_rn(Yz, __dmul_rn(__dmul_rn(0.5, __dadd_rn(zp, zn)), ts_ms));
                xp = xn; yp = yn; zp = zn;
            }
        }
        const int si = step + 1;
        if (active && si % d.steps_per_h == 0) {
            const int j = si / d.steps_per_h;
            Yo[3 * j] = Yx; Yo[3 * j + 1] = Yy; Yo[3 * j + 2] = Yz;
            It[j] = (int8_t)inside;
            if (inside) atomicAdd(reinterpret_cast<unsigned long long*>(&d.occupancy[(size_t)job.slot * d.n_grid + j]), 1ull);
        }
    }
    if (!active) return;
    uint64_t* cnt = d.counters + (size_t)job.slot * MADI_CNT_N;
    atomicAdd(reinterpret_cast<unsigned long long*>(&cnt[MADI_CNT_WALKERS]), 1ull);
    if (escaped) atomicAdd(reinterpret_cast<unsigned long long*>(&cnt[MADI_CNT_ESCAPED]), 1ull);
    if (cerr) atomicAdd(reinterpret_cast<unsigned long long*>(&cnt[MADI_CNT_CLASSIFIER_ERROR]), 1ull);
    atomicAdd(reinterpret_cast<unsigned long long*>(&cnt[MADI_CNT_FULL]), (unsigned long long)n_full);
    atomicAdd(reinterpret_cast<unsigned long long*>(&cnt[MADI_CNT_CROSS_ACCEPT]), (unsigned long long)n_acc);
    atomicAdd(reinterpret_cast<unsigned long long*>(&cnt[MADI_CNT_CROSS_REJECT]), (unsigned long long)n_rej);
    const int8_t i0 = It[0];
    if (i0) atomicAdd(reinterpret_cast<unsigned long long*>(&d.occupancy[(size_t)job.slot * d.n_grid]), 1ull);
}

// ---------------------------------------------------------------------------
// Column reduction from stored Y (replaces _reduce_kernel, madi/walker_gpu.py:
// 658-695, which re-reads Y once per column).  A CTA takes a block of
// REDUCE_COLS columns and a range of walkers.  Consecutive columns with the same
// (jd, jD, js) form a run (the b values of one pair): per walker and axis
// dM = Y[jd] + Y[jD] - Y[js] (the reference's operation order) is computed once
// per run into shared memory and every thread adds cos / sin(coef * dM) of its
// columns.
//
// Bound: the fp64 pipe retires about two lanes per SM and cycle, so a library
// sincos (~35 fp64 operations) made this kernel 303 ms for 31,125 columns x
// 50,000 walkers.  Here a term costs one fp64 operation,
//   r = coef / 2 pi * dM + 1.5 * 2^8 + 2^-13  (fma),
// which leaves the phase in turns modulo 1 in the low 44 mantissa bits: the
// upper 12 choose a table entry (cos, sin of i / 4096 turn in 2^-48 fixed
// point) and the lower 32 the offset x, |x| <= 2^-13 turn.  The addition
// formulas with cos x = 1 - e, sin x = x - x^3 / 6 run in 32 x 32 -> 64 bit
// integer products on the int pipe, terms rounded to 2^-40.  Emulated against
// extended precision: at most 1.8e-12 a term, 4e-13 rms, sums over 1.5e5 terms
// within 2e-10 rms for phases spread over 1e-4 to 50 rad and exact for phase 0.
// A CTA's sums are integers in 2^-48; each is rounded once to 2^-q, the finest
// unit in which 3 n_walkers fits 63 bits, and added to the column's total, so the
// result does not depend on scheduling (bit-identical from run to run).
// Measured at 31,125 columns x 50,000 walkers: 12.0 ms (fp64 pipe 72 % busy);
// error against 64 bits 1.6e-14 of the sums' norm, 3.0e-14 before.
// A chunk of walkers with any |phase| >= 127 turns (or a NaN) goes through
// sincos() in fp64 instead.
// ---------------------------------------------------------------------------
constexpr int REDUCE_CPT = 2;                                // columns per thread
constexpr int REDUCE_COLS = 1024;                            // columns per CTA, at most
constexpr int REDUCE_TAB = 4096;                             // table entries per turn
constexpr int REDUCE_Q = 48;                                 // fraction bits of a CTA's sums
constexpr int REDUCE_WALKERS = 8192;                         // walkers per CTA: 3 * 2^13 * 2^48 < 2^63
constexpr int REDUCE_DM_BYTES = 39424;                       // dM of one walker for 1,024 runs, and more
// table + run triples (uint16 x 3) + largest |coef| of each run + dM: two CTAs an SM
constexpr int REDUCE_SMEM = REDUCE_TAB * 16 + REDUCE_COLS * 6 + REDUCE_COLS * 4 + REDUCE_DM_BYTES;
static_assert(REDUCE_DM_BYTES >= REDUCE_COLS * 24, "one walker's dM must fit");

// cos and sin of one phase, given r = turns + 384 + 2^-13, added to (ac, as).
// Every product is rounded to nearest: a phase of 0 adds exactly (1, 0).
constexpr double REDUCE_MAGIC = 384.0 + 0x1p-13;             // half a table step: the floor of r is the nearest entry
// A table value in 2^-31 (+1 saturates).
MADI_DEV int q31(long long v) {
    const int hi = (int)(v >> 32);
    return hi == 1 << (REDUCE_Q - 32) ? 0x7fffffff : (int)__funnelshift_r((unsigned)v, (unsigned)hi, REDUCE_Q - 31);
}

MADI_DEV void add_cos_sin(double r, const longlong2* tab, long long& ac, long long& as) {
    const int hi = __double2hiint(r), lo = __double2loint(r);
    const longlong2 cs = tab[hi & (REDUCE_TAB - 1)];
    const int x = lo ^ (int)0x80000000;                      // offset from the entry, 2^-44 turn
    const int xx = __mulhi(x, x);
    // 1 - cos(2 pi x) in 2^-51: 2^31 2 pi^2 / 16, less 2.9e-8 of it for the mean of the x^4 term
    const int e = (int)__umulhi((unsigned)xx, 0x9DE9E600u);
    const int e3 = __mulhi(xx, 1685);                        // a third of it in 2^-32
    const int xs = x - (int)(((long long)x * e3 + 0x80000000ll) >> 32);
    const int X = (int)(((long long)xs * 0x6487ED51 + 0x40000000ll) >> 31);   // sin(2 pi x) in 2^-41: 2 pi 2^28
    const int c = q31(cs.x), s = q31(cs.y);
    const int dc = -(int)(((long long)s * X + 0x80000000ll) >> 32) - ((__mulhi(c, e) + 512) >> 10);
    const int ds = (int)(((long long)c * X + 0x80000000ll) >> 32) - ((__mulhi(s, e) + 512) >> 10);
    ac += cs.x + (long long)dc * 256;
    as += cs.y + (long long)ds * 256;
}

template <int THREADS>
__global__ void __launch_bounds__(THREADS, 2) reduce_Y_kernel(const double* __restrict__ Y, int64_t n_walkers,
                                                              int n_grid, int64_t per_block,
                                                              const int32_t* __restrict__ jd,
                                                              const int32_t* __restrict__ jD,
                                                              const int32_t* __restrict__ js,
                                                              const double* __restrict__ coef, int n_cols,
                                                              int shift, unsigned long long* accum) {
    extern __shared__ __align__(16) unsigned char rsm[];
    longlong2* tab = reinterpret_cast<longlong2*>(rsm);
    uint16_t* run = reinterpret_cast<uint16_t*>(rsm + REDUCE_TAB * 16);                          // [runs][3]
    int* run_max = reinterpret_cast<int*>(rsm + REDUCE_TAB * 16 + REDUCE_COLS * 6);              // |turns per dM|
    double* dM = reinterpret_cast<double*>(rsm + REDUCE_TAB * 16 + REDUCE_COLS * 10);            // [walkers][runs][3]
    __shared__ int seg[REDUCE_COLS / 32 + 1];
    const int tid = threadIdx.x, lane = tid & 31;
    constexpr int COLS = THREADS * REDUCE_CPT;
    static_assert(COLS <= REDUCE_COLS && COLS / 32 <= 32, "run table and segment scan");
    const int col0 = blockIdx.x * COLS;
    const int cols = min(COLS, n_cols - col0);
    // ---- table: cos / sin of i / 4096 turn from 32 coarse and 32 fine
    // angles of the first quadrant (one complex product), mirrored ----
    double2* cf = reinterpret_cast<double2*>(dM);
    if (tid < 64) {
        const double turn = tid < 32 ? tid / 128.0 : (tid - 32) / 4096.0;
        double sn, cn;
        sincospi(2.0 * turn, &sn, &cn);
        cf[tid] = make_double2(cn, sn);
    }
    __syncthreads();
    for (int i = tid; i < REDUCE_TAB / 4; i += THREADS) {
        const double2 u = cf[i >> 5], v = cf[32 + (i & 31)];
        const long long c = __double2ll_rn((u.x * v.x - u.y * v.y) * (double)(1ll << REDUCE_Q));
        const long long s = __double2ll_rn((u.y * v.x + u.x * v.y) * (double)(1ll << REDUCE_Q));
        tab[i] = make_longlong2(c, s);
        tab[i + REDUCE_TAB / 4] = make_longlong2(-s, c);
        tab[i + REDUCE_TAB / 2] = make_longlong2(-c, -s);
        tab[i + 3 * REDUCE_TAB / 4] = make_longlong2(s, -c);
    }
    // ---- runs of equal (jd, jD, js) among this block's columns ----
    for (int i = tid; i < COLS; i += THREADS) run_max[i] = 0;
    double pc[REDUCE_CPT];                                   // turns per dM
    int my_run[REDUCE_CPT];
    long long ac[REDUCE_CPT], as[REDUCE_CPT];
#pragma unroll
    for (int k = 0; k < REDUCE_CPT; ++k) {
        const int i = k * THREADS + tid;
        const int col = col0 + i;
        const bool live = i < cols;
        const bool head = live && (i == 0 || jd[col] != jd[col - 1] || jD[col] != jD[col - 1] || js[col] != js[col - 1]);
        const unsigned heads = __ballot_sync(MADI_FULL, head);
        if (lane == 0) seg[i >> 5] = __popc(heads);
        my_run[k] = __popc(heads & (0xffffffffu >> (31 - lane))) - 1;
        pc[k] = live ? __dmul_rn(coef[col], 0.15915494309189535) : 0.0;
        ac[k] = as[k] = 0;
    }
    __syncthreads();
    if (tid < 32) {
        int v = lane < COLS / 32 ? seg[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(MADI_FULL, v, o);
            if (lane >= o) v += u;
        }
        __syncwarp();
        seg[lane + 1] = v;
        if (lane == 0) seg[0] = 0;
    }
    __syncthreads();
    const int runs = seg[COLS / 32];
    const int kmax = (cols + THREADS - 1) / THREADS;
#pragma unroll
    for (int k = 0; k < REDUCE_CPT; ++k) {
        const int i = k * THREADS + tid;
        my_run[k] += seg[i >> 5];
        if (i < cols) {
            const int col = col0 + i;
            run[3 * my_run[k]] = (uint16_t)(3 * jd[col]);    // the same values from every column of the run
            run[3 * my_run[k] + 1] = (uint16_t)(3 * jD[col]);
            run[3 * my_run[k] + 2] = (uint16_t)(3 * js[col]);
            atomicMax(&run_max[my_run[k]], __float_as_int(fabsf((float)pc[k])));
        } else {
            my_run[k] = 0;                                   // dead columns add a phase of 0 nobody reads
        }
    }
    __syncthreads();
    const int row_len = n_grid * 3, r3 = runs * 3;
    const int wt = min(32, REDUCE_DM_BYTES / (r3 * 8));
    const int64_t w0 = (int64_t)blockIdx.y * per_block;
    const int64_t w1 = min(n_walkers, w0 + per_block);
    for (int64_t wb = w0; wb < w1; wb += wt) {
        const int nw = (int)min((int64_t)wt, w1 - wb);
        bool big = false;
        for (int i = tid; i < nw * r3; i += THREADS) {
            const int w = i / r3, j = i - w * r3, t = j / 3, ax = j - 3 * t;
            const double* y = Y + (size_t)(wb + w) * row_len + ax;
            const double dm = __dsub_rn(__dadd_rn(y[run[3 * t]], y[run[3 * t + 1]]), y[run[3 * t + 2]]);
            dM[i] = dm;
            big |= !(fabsf((float)dm) * __int_as_float(run_max[t]) < 127.0f);
        }
        if (!__syncthreads_or(big)) {
            for (int w = 0; w < nw; ++w) {
#pragma unroll
                for (int k = 0; k < REDUCE_CPT; ++k) {
                    if (k >= kmax) break;
                    const double* m = dM + w * r3 + 3 * my_run[k];
#pragma unroll
                    for (int ax = 0; ax < 3; ++ax) add_cos_sin(__fma_rn(pc[k], m[ax], REDUCE_MAGIC), tab, ac[k], as[k]);
                }
            }
        } else {
#pragma unroll
            for (int k = 0; k < REDUCE_CPT; ++k) {
                const int i = k * THREADS + tid;
                if (i >= cols) break;
                const double co = coef[col0 + i];
                double cs = 0.0, sn = 0.0;
                for (int j = 0; j < nw * 3; ++j) {
                    double s, c;
                    sincos(__dmul_rn(co, dM[j / 3 * r3 + 3 * my_run[k] + j % 3]), &s, &c);
                    cs += c;
                    sn += s;
                }
                ac[k] += __double2ll_rn(cs * (double)(1ll << REDUCE_Q));
                as[k] += __double2ll_rn(sn * (double)(1ll << REDUCE_Q));
            }
        }
        __syncthreads();                                     // dM is rewritten
    }
    const long long half = shift > 0 ? 1ll << (shift - 1) : 0ll;
#pragma unroll
    for (int k = 0; k < REDUCE_CPT; ++k) {
        const int i = k * THREADS + tid;
        if (i < cols && w1 > w0) {
            atomicAdd(&accum[col0 + i], (unsigned long long)((ac[k] + half) >> shift));
            atomicAdd(&accum[n_cols + col0 + i], (unsigned long long)((as[k] + half) >> shift));
        }
    }
}

__global__ void reduce_Y_finish_kernel(const long long* accum, int n_cols, double unit, double* cos_sum, double* sin_sum) {
    const int col = blockIdx.x * blockDim.x + threadIdx.x;
    if (col >= n_cols) return;
    cos_sum[col] = (double)accum[col] * unit;
    sin_sum[col] = (double)accum[n_cols + col] * unit;
}

}  // namespace madi

using namespace madi;

extern "C" int64_t madi_walk_smem_bytes(int32_t stage_bytes, int32_t tile_walkers, int32_t n_grid) {
    // the fused layout of fused_smem() at the largest output shape (8 pairs)
    const int64_t n_out = (int64_t)MADI_MAX_PAIRS * MADI_MAX_B * MADI_MAX_DIRS;
    return (int64_t)((stage_bytes + 15) & ~15) + 16ll * n_out + 12ll * ((n_grid + 3) & ~3) +
           (24ll + FC_BYTES_PER_WALKER + 4 * (3 + 3 * MADI_MAX_PAIRS) + 12) * tile_walkers;
}

static int64_t fused_smem(const madi_walk_desc* d, int np, int threads) {
    const int64_t n_out = (int64_t)d->n_pairs * d->n_b * d->n_dirs;
    return (int64_t)d->stage_smem + 16ll * n_out + 12ll * ((d->n_grid + 3) & ~3) +
           (24 + FC_BYTES_PER_WALKER + 4 * (3 + 3 * np) + 12) * threads;
}

// Walkers of a launch that leaves the chip idle go 16 or 8 to a warp where the
// caller says that the launch has it to itself (MADI_WALK_ALONE).  A step is a
// chain of ~2,200 cycles for a warp alone on its scheduler: 416 of them draw the
// random numbers, which the free lanes then do for later steps (2 or 4 pairs at
// once), and ~700 are facet passes, taken if any lane of the warp misses its cache:
// fewer lanes, fewer passes.  10,000 walkers x 4,600 steps in a 64-cell box, 32 / 16
// / 8 to a warp: 5.85 / 5.24 / 4.84 ms; 1,000: 5.80 / 5.03 / 4.42.
//
// The line is half a wave of the CTAs an SM holds.  Past one wave the second costs
// more than this saves (40,000 walkers: 7.0 / 11.3 ms), and a walk that comes along
// after all needs room: two launches of 20,000, the first in a full wave of its own,
// take 12.6 ms, both 32 to a warp 7.1 ms.  Two launches that both took lane groups
// unasked made 9.3 ms of what 32 to a warp do in 6.3 (10,000 walkers each), eight
// 27.7 ms of 12.8.
constexpr int SPREAD_CTAS = 3;                   // resident on an SM: 168 registers a thread, no spills
static bool walk_alone(const madi_walk_desc* d) { return d->min_blocks > 0 && (d->min_blocks & MADI_WALK_ALONE); }
static bool two_blocks(const madi_walk_desc* d) { return d->min_blocks - (walk_alone(d) ? MADI_WALK_ALONE : 0) >= 2; }

static int spread_of(const madi_walk_desc* d, int64_t smem) {
    if (!walk_alone(d)) return 0;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 0;
    const int64_t ctas = sms * std::min<int64_t>(SPREAD_CTAS, 227 * 1024 / (smem + 1024));
    for (int spread = 2; spread > 0; --spread) {
        const int64_t threads = (int64_t)d->n_tiles * d->tile_walkers << spread;
        if (((d->tile_walkers << spread) % SPREAD_THREADS) == 0 && 2 * threads <= ctas * SPREAD_THREADS) return spread;
    }
    return 0;
}

template <int OUT, bool PER, int NP, int MINB, bool SPREAD>
static madi_status launch_f32(const madi_walk_desc* d, int spread, cudaStream_t s) {
    auto k = walk_f32_kernel<OUT, PER, NP, MINB, SPREAD>;
    const int threads = SPREAD ? SPREAD_THREADS : d->tile_walkers;
    const int64_t sm = fused_smem(d, NP, threads);
    if (sm > 227 * 1024) return host::fail(MADI_ERR_CAPACITY, "walker shared memory %lld B exceeds 227 KB", (long long)sm);
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (SPREAD && e == cudaSuccess) {
        // as much shared memory an SM as four CTAs of a launch without lane groups
        // need: with less, such a launch waits for this one's SMs to drain before it
        // gets any (10,000 walkers beside 10,000 of these: 12.3 ms, 6.9 ms so)
        const int64_t percent = (4 * (sm + 1024) * 100 + 228 * 1024 - 1) / (228 * 1024);
        e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, (int)std::min<int64_t>(percent, 100));
    }
    if (e != cudaSuccess) return host::cuda_fail(e, "cudaFuncSetAttribute(walker)");
    const int parts = SPREAD ? (d->tile_walkers << spread) / SPREAD_THREADS : 1;
    const int blocks = (d->grid_blocks > 0 ? d->grid_blocks : d->n_tiles) * parts;
    k<<<blocks, threads, (size_t)sm, s>>>(*d, spread);
    e = cudaGetLastError();
    if (e != cudaSuccess) return host::cuda_fail(e, "walker launch");
    return MADI_OK;
}

template <int OUT, bool PER, int NP>
static madi_status launch_spread(const madi_walk_desc* d, cudaStream_t s) {
    const int spread = spread_of(d, fused_smem(d, NP, SPREAD_THREADS));
    if (spread) return launch_f32<OUT, PER, NP, SPREAD_CTAS, true>(d, spread, s);
    return two_blocks(d) ? launch_f32<OUT, PER, NP, 2, false>(d, 0, s) : launch_f32<OUT, PER, NP, 1, false>(d, 0, s);
}

template <int OUT, bool PER>
static madi_status launch_np(const madi_walk_desc* d, cudaStream_t s) {
    if (OUT == MADI_OUT_FUSED && d->n_pairs > 4) return launch_spread<OUT, PER, 8>(d, s);
    return launch_spread<OUT, PER, 4>(d, s);
}

template <int OUT, bool PER>
static const void* kernel_for(const madi_walk_desc* d) {
    const bool two = two_blocks(d);
    if (OUT == MADI_OUT_FUSED && d->n_pairs > 4)
        return two ? (const void*)walk_f32_kernel<OUT, PER, 8, 2, false> : (const void*)walk_f32_kernel<OUT, PER, 8, 1, false>;
    return two ? (const void*)walk_f32_kernel<OUT, PER, 4, 2, false> : (const void*)walk_f32_kernel<OUT, PER, 4, 1, false>;
}

extern "C" int32_t madi_walk_blocks_per_sm(const madi_walk_desc* d) {
    if (!d || d->tile_walkers <= 0) return 0;
    const bool per = d->boundary == MADI_BOUNDARY_PERIODIC;
    const void* k = d->out_mode == MADI_OUT_FUSED
        ? (per ? kernel_for<MADI_OUT_FUSED, true>(d) : kernel_for<MADI_OUT_FUSED, false>(d))
        : (per ? kernel_for<MADI_OUT_Y, true>(d) : kernel_for<MADI_OUT_Y, false>(d));
    const bool big = d->out_mode == MADI_OUT_FUSED && d->n_pairs > 4;
    const int64_t sm = fused_smem(d, big ? 8 : 4, d->tile_walkers);
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm) != cudaSuccess) return 0;
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, d->tile_walkers, (size_t)sm) != cudaSuccess) return 0;
    return n;
}

extern "C" madi_status madi_walk(const madi_walk_desc* d, void* stream) {
    host::clear_error();
    if (!d) return host::fail(MADI_ERR_INVALID, "null walk descriptor");
    if (d->n_jobs <= 0 || d->n_geoms <= 0 || !d->jobs || !d->geoms)
        return host::fail(MADI_ERR_INVALID, "walk needs at least one job and one geometry");
    if (d->n_steps < 0 || d->steps_per_h <= 0 || d->n_grid <= 0 || d->n_grid > MADI_MAX_GRID)
        return host::fail(MADI_ERR_INVALID, "bad step grid (n_steps=%d steps_per_h=%d n_grid=%d)",
                          d->n_steps, d->steps_per_h, d->n_grid);
    if (d->n_steps / d->steps_per_h + 1 > d->n_grid)
        return host::fail(MADI_ERR_INVALID, "n_grid too small for n_steps / steps_per_h");
    if (!d->counters || !d->occupancy) return host::fail(MADI_ERR_INVALID, "counters and occupancy are required");
    if (d->rng == MADI_RNG_STREAM && (!d->init || !d->incr || !d->unif))
        return host::fail(MADI_ERR_INVALID, "stream replay needs init / incr / unif");
    // a replay stream brings its own steps
    if (d->rng == MADI_RNG_PHILOX && !std::isfinite(d->precision == 32 ? (double)(float)d->sigma : d->sigma))
        return host::fail(MADI_ERR_INVALID, "walk: sigma %g is not a finite step", d->sigma);
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (d->precision == 64) {
        if (d->n_jobs != 1) return host::fail(MADI_ERR_UNSUPPORTED, "fp64 walker walks one job");
        if (!d->Y || !d->inside_trace) return host::fail(MADI_ERR_INVALID, "fp64 walker writes Y and inside_trace");
        // The job is read on the device; the host only needs its walker count, passed as n_tiles * 128 bound.
        const int blocks = d->n_tiles;
        walk_f64_kernel<<<blocks, F64_THREADS, 0, s>>>(*d);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return host::cuda_fail(e, "fp64 walker launch");
        return MADI_OK;
    }
    if (d->precision != 32) return host::fail(MADI_ERR_INVALID, "precision must be 32 or 64");
    if (d->tile_walkers <= 0 || d->tile_walkers > 256 || (d->tile_walkers & 31))
        return host::fail(MADI_ERR_INVALID, "tile_walkers must be a multiple of 32 in [32, 256]");
    if (d->grid_blocks > 0 && !d->work_counter) return host::fail(MADI_ERR_INVALID, "persistent launch needs a zeroed work counter");
    if (d->out_mode == MADI_OUT_FUSED) {
        if (d->n_pairs < 1 || d->n_pairs > MADI_MAX_PAIRS || d->n_b < 1 || d->n_b > MADI_MAX_B ||
            d->n_dirs < 1 || d->n_dirs > MADI_MAX_DIRS)
            return host::fail(MADI_ERR_UNSUPPORTED, "fused epilogue holds <= %d pairs, <= %d b, <= %d dirs",
                              MADI_MAX_PAIRS, MADI_MAX_B, MADI_MAX_DIRS);
        if ((int64_t)d->n_pairs * d->n_b * d->n_dirs > 2048)
            return host::fail(MADI_ERR_UNSUPPORTED, "fused epilogue holds <= 2048 (column, direction) outputs");
        if (!d->accum) return host::fail(MADI_ERR_INVALID, "fused output needs accum");
        for (int p = 0; p < d->n_pairs; ++p)
            if (d->pair_jd[p] < 0 || d->pair_jD[p] < 0 || d->pair_js[p] < 0 || d->pair_jd[p] >= d->n_grid ||
                d->pair_jD[p] >= d->n_grid || d->pair_js[p] >= d->n_grid)
                return host::fail(MADI_ERR_INVALID, "pair grid index out of range");
    } else if (d->out_mode == MADI_OUT_Y) {
        if (!d->Y || !d->inside_trace) return host::fail(MADI_ERR_INVALID, "Y output needs Y and inside_trace");
    } else {
        return host::fail(MADI_ERR_INVALID, "unknown out_mode");
    }
    if (d->stage_smem < 0 || (d->stage_smem & 15)) return host::fail(MADI_ERR_INVALID, "stage_smem must be a multiple of 16");
    const bool per = d->boundary == MADI_BOUNDARY_PERIODIC;
    if (d->out_mode == MADI_OUT_FUSED)
        return per ? launch_np<MADI_OUT_FUSED, true>(d, s) : launch_np<MADI_OUT_FUSED, false>(d, s);
    return per ? launch_np<MADI_OUT_Y, true>(d, s) : launch_np<MADI_OUT_Y, false>(d, s);
}

extern "C" int64_t madi_reduce_Y_scratch_bytes(int32_t n_cols) {
    return n_cols > 0 ? 16ll * n_cols : 0;
}

extern "C" madi_status madi_reduce_Y(const double* Y, int64_t n_walkers, int32_t n_grid, const int32_t* jd,
                                     const int32_t* jD, const int32_t* js, const double* coef, int32_t n_cols,
                                     double* cos_sum, double* sin_sum, void* scratch, int64_t scratch_bytes,
                                     void* stream) {
    host::clear_error();
    if (!Y || !jd || !jD || !js || !coef || !cos_sum || !sin_sum || n_walkers < 0 || n_grid <= 0 ||
        n_grid > MADI_MAX_GRID || n_cols < 0)
        return host::fail(MADI_ERR_INVALID, "bad reduce_Y arguments");
    if (n_cols == 0) return MADI_OK;
    if (!scratch || scratch_bytes < madi_reduce_Y_scratch_bytes(n_cols))
        return host::fail(MADI_ERR_CAPACITY, "reduce_Y: scratch %lld < %lld bytes", (long long)scratch_bytes,
                          (long long)madi_reduce_Y_scratch_bytes(n_cols));
    if ((reinterpret_cast<uintptr_t>(scratch) & 7) != 0) return host::fail(MADI_ERR_INVALID, "reduce_Y: scratch must be 8-byte aligned");
    // the fixed-point column totals hold 3 n_walkers 2^32 < 2^63
    if (n_walkers > 500000000ll) return host::fail(MADI_ERR_UNSUPPORTED, "reduce_Y: at most 5e8 walkers");
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    unsigned long long* accum = static_cast<unsigned long long*>(scratch);
    cudaError_t e = cudaMemsetAsync(accum, 0, (size_t)madi_reduce_Y_scratch_bytes(n_cols), s);
    if (e != cudaSuccess) return host::cuda_fail(e, "reduce_Y memset");
    // fraction bits of the column totals: 3 n_walkers 2^q < 2^63
    int q = REDUCE_Q;
    while (3.0 * (double)n_walkers * std::ldexp(1.0, q) >= 0x1p63) --q;
    if (n_walkers > 0) {
        // 512 threads hide the chain of a term better (31,125 columns x 50,000
        // walkers: 12.0 ms against 13.0 ms at 256 threads x 4 columns); up to 512
        // columns, 256 threads leave fewer of them idle (200 columns: 0.16 ms
        // against 0.24 ms).
        const int threads = n_cols <= 256 * REDUCE_CPT ? 256 : 512;
        const auto kernel = threads == 256 ? reduce_Y_kernel<256> : reduce_Y_kernel<512>;
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, REDUCE_SMEM);
        if (e != cudaSuccess) return host::cuda_fail(e, "reduce_Y attribute");
        int dev = 0, sms = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        const int gx = (n_cols + threads * REDUCE_CPT - 1) / (threads * REDUCE_CPT);
        // Whole waves of two CTAs an SM; more waves even out the last one as long
        // as a CTA keeps enough walkers to pay for its table (~3 us).
        int64_t gy = 1;
        for (int waves = 1; waves <= 4; waves *= 2) {
            const int64_t y = std::max<int64_t>(1, (int64_t)waves * 2 * sms / gx);
            if (waves == 1 || n_walkers / y >= 64) gy = y;
        }
        int64_t per = std::min<int64_t>((n_walkers + gy - 1) / gy, REDUCE_WALKERS);
        gy = (n_walkers + per - 1) / per;
        kernel<<<dim3((unsigned)gx, (unsigned)gy), threads, REDUCE_SMEM, s>>>(
            Y, n_walkers, n_grid, per, jd, jD, js, coef, n_cols, REDUCE_Q - q, accum);
        e = cudaGetLastError();
        if (e != cudaSuccess) return host::cuda_fail(e, "reduce_Y launch");
    }
    reduce_Y_finish_kernel<<<(n_cols + 255) / 256, 256, 0, s>>>(reinterpret_cast<const long long*>(accum), n_cols,
                                                                std::ldexp(1.0, -q), cos_sum, sin_sum);
    e = cudaGetLastError();
    if (e != cudaSuccess) return host::cuda_fail(e, "reduce_Y finish");
    return MADI_OK;
}

// ---------------------------------------------------------------------------
// Allocation-free walk.  The persistent walker needs one zeroed 32-bit tile
// counter besides its inputs and outputs; this entry point keeps it in a
// file-scope device array instead of a caller buffer, so the caller allocates
// nothing for it.  The array is 256 bytes (one word used), lives on every GPU
// that loads this library until the process exits, and is shared by all calls:
// each call clears the word on its own stream before walking, and two calls
// that overlap on the GPU race on it.
// ---------------------------------------------------------------------------
#include <mutex>

#define MADI_WALK_STATIC_SCRATCH_WORDS 64
static __device__ __align__(256) uint32_t g_walk_static_scratch[MADI_WALK_STATIC_SCRATCH_WORDS];

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_scratch_mu;
uint32_t* g_scratch_addr[kMaxDevices] = {};

// Device address of the static scratch on the current device.  The first call
// on a device resolves it with cudaGetSymbolAddress (that device current) and
// caches it.
madi_status static_scratch(uint32_t** out) {
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return host::cuda_fail(e, "cudaGetDevice");
    if (dev < 0 || dev >= kMaxDevices) return host::fail(MADI_ERR_UNSUPPORTED, "device ordinal %d beyond %d", dev, kMaxDevices);
    std::lock_guard<std::mutex> lock(g_scratch_mu);
    if (!g_scratch_addr[dev]) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_walk_static_scratch);
        if (e != cudaSuccess) return host::cuda_fail(e, "cudaGetSymbolAddress(walk scratch)");
        g_scratch_addr[dev] = static_cast<uint32_t*>(p);
    }
    *out = g_scratch_addr[dev];
    return MADI_OK;
}
}  // namespace

extern "C" madi_status madi_walk_batched(const madi_walk_desc* desc, void* stream) {
    host::clear_error();
    if (!desc) return host::fail(MADI_ERR_INVALID, "walk_batched: null descriptor");
    if (desc->precision != 32) return host::fail(MADI_ERR_INVALID, "walk_batched: fp32 walkers only");
    madi_walk_desc d = *desc;
    if (d.grid_blocks <= 0) {
        int dev = 0, sms = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        const int32_t bps = madi_walk_blocks_per_sm(&d);
        if (bps <= 0) return host::fail(MADI_ERR_CUDA, "walk_batched: no resident block fits this descriptor");
        d.grid_blocks = (int32_t)std::min<int64_t>((int64_t)sms * bps, std::max<int64_t>(d.n_tiles, 1));
    }
    return madi_walk(&d, stream);
}

extern "C" madi_status madi_walk_noalloc(const madi_walk_desc* desc, void* stream) {
    host::clear_error();
    if (!desc) return host::fail(MADI_ERR_INVALID, "null walk descriptor");
    const int64_t handed_out = (int64_t)desc->n_tiles + (desc->grid_blocks > 0 ? desc->grid_blocks : 0);
    if (handed_out >= 0x7FFFFFFFll)
        return host::fail(MADI_ERR_CAPACITY,
                          "walk_noalloc: %lld tiles + CTAs exceed the static scratch counter (max %d)",
                          (long long)handed_out, 0x7FFFFFFF - 1);
    uint32_t* counter = nullptr;
    madi_status st = static_scratch(&counter);
    if (st != MADI_OK) return st;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const cudaError_t e = cudaMemsetAsync(counter, 0, sizeof(uint32_t), s);
    if (e != cudaSuccess) return host::cuda_fail(e, "cudaMemsetAsync(walk scratch)");
    madi_walk_desc d = *desc;
    d.work_counter = counter;
    return madi_walk(&d, stream);
}
