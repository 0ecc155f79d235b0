// kernels.cu -- sm_103a counting kernels.
//
// All kernels are persistent: a grid of (SM count x resident CTAs) draws work
// from a device counter.  Tile kernels: a unit names one spatial tile (<= 64
// points) of roles B and C and a set of A tiles, found by the planner kernels
// from the views' tile boxes; the CTA stages the tiles' points in shared
// memory, computes the side lengths of the tile pairs once (exactly as the
// reference does), and then walks the triangles with one warp per point of
// role A, a loop over role B and the 32 lanes spanning role C.  Neighbour-list
// kernels: a warp or pipeline takes one point at a time, gathers the points
// near it and counts their pairs.  Counts go to shared histograms (32-bit)
// that are flushed with 64-bit global atomics when the histogram changes,
// before they can run over, and at exit.
//
// Exactness: side lengths and their bins are computed with IEEE
// round-to-nearest intrinsics in the reference's operation order, so they equal
// the reference's floats.  The triangle-parametrization fast path then works
// with approximate reciprocals/arc cosines and sends every triangle whose q or
// theta value lies within a bounded guard band of a bin edge to a recheck
// queue; the recheck kernel recomputes those triangles with the reference's
// exact arithmetic (including glibc's acosf through an exception table).
#include <stdint.h>
#include <limits.h>
#include <math.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "../../include/tpcf.h"
#include "engine.h"
#include "exact_acos.h"
#include "plan_bounds.h"

namespace tpcf {

// ---------------------------------------------------------------------------
// Exact reference arithmetic.  FOps<false>: IEEE float intrinsics (never
// contracted).  FOps<true>: each float operation computed in FP64 and rounded
// to float -- identical results for + - * / sqrt (double rounding is innocuous
// when the wide format has at least 2p+2 bits, Figueroa 1995).
template <bool FP64>
struct FOps;
template <>
struct FOps<false> {
    static __device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
    static __device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
    static __device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
    static __device__ __forceinline__ float div(float a, float b) { return __fdiv_rn(a, b); }
    static __device__ __forceinline__ float sqrt(float a) { return __fsqrt_rn(a); }
};
template <>
struct FOps<true> {
    static __device__ __forceinline__ float add(float a, float b) { return __double2float_rn(__dadd_rn(a, b)); }
    static __device__ __forceinline__ float sub(float a, float b) { return __double2float_rn(__dsub_rn(a, b)); }
    static __device__ __forceinline__ float mul(float a, float b) { return __double2float_rn(__dmul_rn(a, b)); }
    static __device__ __forceinline__ float div(float a, float b) { return __double2float_rn(__ddiv_rn(a, b)); }
    static __device__ __forceinline__ float sqrt(float a) { return __double2float_rn(__dsqrt_rn(a)); }
};

// |p0 - p1| as the reference computes it: sqrt((dx*dx + dy*dy) + dz*dz) in
// float (src/3pcf_C_version.cc:57-60, src/3pcf_C_version_triangle_parametrization.cc:119-122,
// src/2pcf_C_version.cc:92-95).  Symmetric in its arguments bit for bit.
template <bool FP64>
__device__ __forceinline__ float ref_dist(float4 a, float4 b) {
    typedef FOps<FP64> F;
    float dx = F::sub(a.x, b.x), dy = F::sub(a.y, b.y), dz = F::sub(a.z, b.z);
    float s = F::mul(dx, dx);
    s = F::add(s, F::mul(dy, dy));
    s = F::add(s, F::mul(dz, dz));
    return F::sqrt(s);
}

// distance_to_bin of the triangle and pair programs
// (src/3pcf_C_version_triangle_parametrization.cc:84-113, src/2pcf_C_version.cc:57-86).
template <bool FP64>
__device__ __forceinline__ int ref_bin_tp(float v, float lo, float hi, int n, int nan_zero) {
    typedef FOps<FP64> F;
    float bw = F::div(F::sub(hi, lo), (float)n);
    if (v < lo) return -999;
    if (v >= hi) return -999;
    if (v != v) return nan_zero ? 0 : INT_MIN;  // int(NaN): aarch64 0, x86-64 INT_MIN
    return __float2int_rz(F::div(F::sub(v, lo), bw));
}

// glibc acosf reproduced exactly: (float)tpcf_acos_d(c) unless c is listed in
// the exception table built on the host from the host's own libm.
__device__ __forceinline__ float acosf_ref(float c, const AcosTable& t) {
    if (!(c >= -1.0f && c <= 1.0f)) return __int_as_float(0x7fc00000);
    float r = __double2float_rn(tpcf_acos_d((double)c));
    uint32_t key = __float_as_uint(c);
    uint32_t lo = t.bucket[key >> 16], hi = t.bucket[(key >> 16) + 1];
    while (lo < hi) {
        uint32_t mid = (lo + hi) >> 1;
        if (t.keys[mid] < key) lo = mid + 1;
        else hi = mid;
    }
    if (lo < t.n && t.keys[lo] == key) r = __uint_as_float(t.vals[lo]);
    return r;
}

// distance() of the triangle program (:116-240) after the side lengths:
// three histogram indices, or -1 for "not counted" (out of range, zero side, or
// an index past the array end, which the reference never prints).
template <bool FP64>
__device__ void tp_exact(float dist0, float dist1, float dist2, const TriParams& p, const AcosTable& t,
                         int out[3]) {
    typedef FOps<FP64> F;
    float shortest, middle, longest;
    if (dist0 > dist1) {
        if (dist0 > dist2) {
            longest = dist0;
            if (dist1 > dist2) { middle = dist1; shortest = dist2; }
            else { middle = dist2; shortest = dist1; }
        } else {
            middle = dist0;
            if (dist1 > dist2) { longest = dist1; shortest = dist2; }
            else { longest = dist2; shortest = dist1; }
        }
    } else {
        if (dist1 > dist2) {
            longest = dist1;
            if (dist0 > dist2) { middle = dist0; shortest = dist2; }
            else { middle = dist2; shortest = dist0; }
        } else {
            middle = dist1; longest = dist2; shortest = dist0;
        }
    }
    float s2 = F::mul(shortest, shortest), m2 = F::mul(middle, middle), l2 = F::mul(longest, longest);
    bool zero = dist0 == 0.f || dist1 == 0.f || dist2 == 0.f;
    float th0 = 0.f, th1 = 0.f;
    for (int k = 0; k < 3; k++) {
        float s, q;
        int i2;
        if (k == 0) {
            s = shortest;
            q = F::div(middle, shortest);
            float c = F::div(F::sub(F::add(s2, m2), l2), F::mul(F::mul(2.f, shortest), middle));
            th0 = __double2float_rn(__ddiv_rn((double)acosf_ref(c, t), 3.14159));
            i2 = ref_bin_tp<FP64>(th0, p.t_lo, p.t_hi, p.T, p.nan_zero);
        } else if (k == 1) {
            s = middle;
            q = F::div(longest, middle);
            float c = F::div(F::sub(F::add(m2, l2), s2), F::mul(F::mul(2.f, middle), longest));
            th1 = __double2float_rn(__ddiv_rn((double)acosf_ref(c, t), 3.14159));
            i2 = ref_bin_tp<FP64>(th1, p.t_lo, p.t_hi, p.T, p.nan_zero);
        } else {
            s = shortest;
            q = F::div(longest, shortest);
            float th2 = __double2float_rn(__dsub_rn(__dsub_rn(1.0, (double)th0), (double)th1));
            i2 = ref_bin_tp<FP64>(th2, p.t_lo, p.t_hi, p.T, p.nan_zero);
        }
        int i0 = ref_bin_tp<FP64>(s, p.s_lo, p.s_hi, p.S, p.nan_zero);
        int i1 = ref_bin_tp<FP64>(q, p.q_lo, p.q_hi, p.Q, p.nan_zero);
        int tot = -1;
        if (!(i0 < 0 || i1 < 0 || i2 < 0) && !zero) {
            long long idx = (long long)p.Q * p.T * i0 + (long long)p.T * i1 + i2;
            if (idx < p.len) tot = (int)idx;
        }
        out[k] = tot;
    }
}

// ---------------------------------------------------------------------------
// The same triangle formulas evaluated in double from the float coordinates,
// acos in double: not the reference's float arithmetic, but the FP64 truth
// the derived correlation function's error is quoted against.  Every
// operation is an explicit round-to-nearest double op (no contraction), so a
// host restatement compiled without FMA contraction agrees except where the
// two acos implementations differ.

__device__ __forceinline__ double geo_dist(float4 a, float4 b) {
    double dx = __dsub_rn((double)a.x, (double)b.x);
    double dy = __dsub_rn((double)a.y, (double)b.y);
    double dz = __dsub_rn((double)a.z, (double)b.z);
    double s = __dmul_rn(dx, dx);
    s = __dadd_rn(s, __dmul_rn(dy, dy));
    s = __dadd_rn(s, __dmul_rn(dz, dz));
    return __dsqrt_rn(s);
}

__device__ __forceinline__ int geo_bin(double v, float lo, float hi, int n, int nan_zero) {
    double bw = __ddiv_rn(__dsub_rn((double)hi, (double)lo), (double)n);
    if (v < (double)lo) return -999;
    if (v >= (double)hi) return -999;
    if (v != v) return nan_zero ? 0 : INT_MIN;
    return __double2int_rz(__ddiv_rn(__dsub_rn(v, (double)lo), bw));
}

__device__ void tp_geom(double d0, double d1, double d2, const TriParams& p, int out[3]) {
    // shortest <= middle <= longest with the reference's tie handling
    double shortest, middle, longest;
    if (d0 > d1) {
        if (d0 > d2) {
            longest = d0;
            if (d1 > d2) { middle = d1; shortest = d2; }
            else { middle = d2; shortest = d1; }
        } else {
            middle = d0;
            if (d1 > d2) { longest = d1; shortest = d2; }
            else { longest = d2; shortest = d1; }
        }
    } else {
        if (d1 > d2) {
            longest = d1;
            if (d0 > d2) { middle = d0; shortest = d2; }
            else { middle = d2; shortest = d0; }
        } else {
            middle = d1; longest = d2; shortest = d0;
        }
    }
    const double s2 = __dmul_rn(shortest, shortest), m2 = __dmul_rn(middle, middle), l2 = __dmul_rn(longest, longest);
    const bool zero = d0 == 0.0 || d1 == 0.0 || d2 == 0.0;
    double c0 = __ddiv_rn(__dsub_rn(__dadd_rn(s2, m2), l2), __dmul_rn(__dmul_rn(2.0, shortest), middle));
    double c1 = __ddiv_rn(__dsub_rn(__dadd_rn(m2, l2), s2), __dmul_rn(__dmul_rn(2.0, middle), longest));
    double th0 = __ddiv_rn(acos(c0), 3.14159), th1 = __ddiv_rn(acos(c1), 3.14159);
    double th2 = __dsub_rn(__dsub_rn(1.0, th0), th1);
    const double sv[3] = {shortest, middle, shortest};
    const double qv[3] = {__ddiv_rn(middle, shortest), __ddiv_rn(longest, middle), __ddiv_rn(longest, shortest)};
    const double tv[3] = {th0, th1, th2};
#pragma unroll
    for (int k = 0; k < 3; k++) {
        int i0 = geo_bin(sv[k], p.s_lo, p.s_hi, p.S, p.nan_zero);
        int i1 = geo_bin(qv[k], p.q_lo, p.q_hi, p.Q, p.nan_zero);
        int i2 = geo_bin(tv[k], p.t_lo, p.t_hi, p.T, p.nan_zero);
        int tot = -1;
        if (!(i0 < 0 || i1 < 0 || i2 < 0) && !zero) {
            long long idx = (long long)p.Q * p.T * i0 + (long long)p.T * i1 + i2;
            if (idx < p.len) tot = (int)idx;
        }
        out[k] = tot;
    }
}

// ---------------------------------------------------------------------------
// Persistent-task plumbing.

constexpr unsigned int FLUSH_EVERY = 256;  // tasks between histogram flushes (u32 safety)
constexpr uint32_t TASK_NONE = 0xFFFFFFFFu;

// A single-tile unit as {slot, tile A, tile B, tile C} (slot TASK_NONE past
// the end) and the points [i0, i1) of tile A it covers; drawn by one thread.
__device__ __forceinline__ uint4 draw_unit(const UnitList& ul, unsigned int* counter, int& i0, int& i1) {
    const unsigned int t = atomicAdd(counter, 1u);
    i0 = 0;
    i1 = TILE;
    if (t >= ul.n || ul.u0 + t >= ul.header->nunits) return make_uint4(TASK_NONE, 0, 0, 0);
    uint4 u = ul.units[ul.u0 + t];
    if (u.x & UNIT_QUARTER) {
        i0 = (int)((u.x >> UNIT_QUARTER_SHIFT) & 3u) * (TILE / 4);
        i1 = i0 + TILE / 4;
    }
    return make_uint4(u.x & UNIT_SLOT_MASK, u.y + (uint32_t)__ffs(ul.masks[ul.u0 + t]) - 1u, u.z, u.w);
}

// Swizzled shared histograms (three-side kernels): bin b of a copy lives at
// word hist_pos(b), its low five bits (the bank) XORed with the next two 5-bit
// groups, so that the lanes of one atomic instruction whose bins differ only
// in higher digits (n^2 i2 + n i1 + i0 with n = 32 puts every lane of a
// three-side row in one bank) spread over the banks.  It permutes each
// aligned group of 32 words, so a copy takes hist_stride(words) words.
__host__ __device__ constexpr int hist_stride(int len) { return (len + 31) & ~31; }
__device__ __forceinline__ unsigned hist_pos(unsigned b) { return b ^ (((b >> 5) ^ (b >> 10)) & 31u); }

// Adds 'copies' shared histograms of len bins (len words apart) into the
// job's 64-bit histogram and clears them.
__device__ __forceinline__ void flush_hist(unsigned int* H, int copies, int len, unsigned long long* g) {
    __syncthreads();
    for (int b = threadIdx.x; b < len; b += blockDim.x) {
        unsigned long long sum = 0;
        for (int c = 0; c < copies; c++) {
            sum += H[c * len + b];
            H[c * len + b] = 0;
        }
        if (sum) atomicAdd(g + b, sum);
    }
    __syncthreads();
}

__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float rsqrt_approx(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// ---------------------------------------------------------------------------
// Planning.  A launch's units of work -- tile triples (or, for the fast
// triangle kernel, a tile pair (B, C) with a mask of up to `window` A tiles)
// that can hold a counted triple -- are found on the device from the views'
// tile boxes: row (job, window of A tiles, tile B) tests every tile C.
//   plan_rows<false>  units of each row, those of each block of rows, and totals;
//   plan_scan         (one CTA) exclusive scan of the blocks' sums, the number of
//                     parts heavy units are cut into, the header;
//   plan_rows<true>   the same tests again, writing each unit to its place (the
//                     two passes have to decide alike: see plan_bounds.h).
// Heavy units (an estimate of their triples above PlanParams::heavy) come
// first, in job order, then the light ones in job order: a CTA flushes its
// histogram when the job changes, and the long units are not left to the end.
// With few of them for the CTAs, each is cut into its A tiles or the quarters
// of those.  (The 40,000 voxel jobs of a 20k-point cone took 22 ms to plan on
// 16 host cores, 0.95M tile triples of 150k points 9.3 ms; both are below 1 ms
// here.)

constexpr int PLAN_WARPS = 8;

// Last job j of [0, n) with off[j] <= t (off[0] <= t; a job without items is
// never the last one), searched 32 ways at a time by a whole warp.
__device__ __forceinline__ int find_job(const uint32_t* __restrict__ off, int n, uint32_t t) {
    const int lane = threadIdx.x & 31;
    int lo = 0, len = n;
    while (len > 1) {
        const int step = (len + 31) / 32;
        const bool le = lane * step < len && off[lo + lane * step] <= t;
        const int k = 31 - __clz(__ballot_sync(0xffffffffu, le) | 1u);
        lo += k * step;
        len = min(step, len - k * step);
    }
    return lo;
}

int plan_blocks(uint64_t nrows, int* rows_per_block) {
    // one row per warp while that leaves the scan few sums, else eight
    const int r = nrows <= 32768 ? PLAN_WARPS : PLAN_WARPS * 8;
    if (rows_per_block) *rows_per_block = r;
    return (int)((nrows + r - 1) / r);
}

template <bool FILL>
__global__ void __launch_bounds__(PLAN_WARPS * 32)
plan_rows(const DevJob* __restrict__ jobs, const uint32_t* __restrict__ row_off, int njobs, uint32_t nrows,
          int rows_per_block, PlanParams pp, uint2* row_cnt, uint2* block_sum, PlanHeader* header, uint4* units,
          uint32_t* masks) {
    __shared__ float4 s_box[PLAN_WARPS][2 * MAX_WINDOW];
    __shared__ float2 s_ab[PLAN_WARPS][MAX_WINDOW];
    __shared__ int s_na[PLAN_WARPS][MAX_WINDOW];
    __shared__ uint2 s_sum[PLAN_WARPS];
    __shared__ unsigned long long s_eval, s_tiles;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned full = 0xffffffffu;
    if (!FILL && threadIdx.x == 0) s_eval = s_tiles = 0ull;
    uint32_t nunits = 0, nheavy = 0, parts = 0;
    if (FILL) {
        nunits = header->nunits;
        if (nunits == 0) return;  // nothing found, or more than the list holds
        parts = header->parts;
        nheavy = block_sum[gridDim.x].x;
    }
    __syncthreads();
    const uint32_t row0 = blockIdx.x * (uint32_t)rows_per_block;
    // consecutive rows of the block go to one warp
    const int per_warp = rows_per_block / PLAN_WARPS;
    uint2 place = make_uint2(0, 0);  // FILL: heavy and light units before this warp's rows
    if (FILL) {
        for (int r = lane; r < warp * per_warp; r += 32)
            if (row0 + r < nrows) {
                const uint2 c = row_cnt[row0 + r];
                place.x += c.x;
                place.y += c.y;
            }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            place.x += __shfl_xor_sync(full, place.x, o);
            place.y += __shfl_xor_sync(full, place.y, o);
        }
        place.x += block_sum[blockIdx.x].x;
        place.y += block_sum[blockIdx.x].y;
    }
    uint2 warp_sum = make_uint2(0, 0);
    unsigned long long eval = 0, tiles = 0;
    for (int rr = 0; rr < per_warp; rr++) {
        const uint32_t row = row0 + (uint32_t)(warp * per_warp + rr);
        if (row >= nrows) break;
        uint2 expect = make_uint2(0, 0);  // FILL: the places after this row's units
        if (FILL) {
            const uint2 c = row_cnt[row];
            if (c.x + c.y == 0u) continue;
            expect = make_uint2(place.x + c.x, place.y + c.y);
        }
        const int slot = find_job(row_off, njobs, row);
        const DevJob& J = jobs[slot];
        const uint32_t l = row - row_off[slot];
        const int ntA = J.ntiles[0], ntB = J.ntiles[1], ntC = J.ntiles[2];
        const int a0 = (int)(l / (uint32_t)ntB) * pp.window, b = (int)(l % (uint32_t)ntB);
        const bool from_a = J.mode & JOB_B_FROM_A, from_b = J.mode & JOB_C_FROM_B;
        const float4 bl = J.box[1][2 * (size_t)b], bh = J.box[1][2 * (size_t)b + 1];
        const int nb = J.tile_start[1][b + 1] - J.tile_start[1][b];
        bool ok = false;
        __syncwarp();
        if (lane < pp.window && a0 + lane < ntA && (!from_a || b >= a0 + lane)) {
            const float4 al = J.box[0][2 * (size_t)(a0 + lane)], ah = J.box[0][2 * (size_t)(a0 + lane) + 1];
            const float2 ab = box_bounds2(al, ah, bl, bh);
            ok = !(ab.x >= pp.lmax2);
            s_box[warp][2 * lane] = al;
            s_box[warp][2 * lane + 1] = ah;
            s_ab[warp][lane] = ab;
            s_na[warp][lane] = J.tile_start[0][a0 + lane + 1] - J.tile_start[0][a0 + lane];
        }
        const unsigned amask = __ballot_sync(full, ok);
        __syncwarp();
        uint2 cnt = make_uint2(0, 0);  // this lane's units of the row
        if (amask) {
            for (int c0 = from_b ? b & ~31 : 0; c0 < ntC; c0 += 32) {
                const int c = c0 + lane;
                const bool in = c < ntC && (!from_b || c >= b);
                float4 cl = make_float4(0.f, 0.f, 0.f, 0.f), ch = cl;
                float2 bc = make_float2(0.f, 0.f);
                bool cand = in;
                if (in) {
                    cl = J.box[2][2 * (size_t)c];
                    ch = J.box[2][2 * (size_t)c + 1];
                    bc = box_bounds2(bl, bh, cl, ch);
                    cand = !(bc.x >= pp.lmax2);
                }
                if (!__any_sync(full, cand)) continue;
                unsigned mask = 0;
                float est = 0.f;
                unsigned n_heavy = 0, n_light = 0;
                if (cand) {
                    const int nc = J.tile_start[2][c + 1] - J.tile_start[2][c];
                    for (unsigned m = amask; m; m &= m - 1u) {
                        const int t = __ffs(m) - 1;
                        const float2 ab = s_ab[warp][t], ac = box_bounds2(s_box[warp][2 * t], s_box[warp][2 * t + 1], cl, ch);
                        if (ac.x >= pp.lmax2 || (pp.tri && !tri_possible(ab, ac, bc, pp))) continue;
                        mask |= 1u << t;
                        if (pp.heavy > 0.f)
                            est = add_estimate(est, (float)s_na[warp][t], (float)nb, (float)nc, ab, ac, bc, pp.r);
                        if (!FILL) {
                            const unsigned long long na = (unsigned)s_na[warp][t], n = (unsigned)nb, k = (unsigned)nc;
                            const bool dij = from_a && a0 + t == b, djk = from_b && b == c;
                            eval += dij && djk ? na * (na - 1) * (na - 2) / 6
                                    : dij      ? na * (na - 1) / 2 * k
                                    : djk      ? na * (n * (n - 1) / 2)
                                               : na * n * k;
                        }
                    }
                    const unsigned n = pp.per_tile ? __popc(mask) : (mask ? 1u : 0u);
                    tiles += __popc(mask);
                    // (without estimates every unit is a heavy one)
                    if (!(pp.heavy > 0.f) || est > pp.heavy) n_heavy = n;
                    else n_light = n;
                }
                if (!FILL) {
                    cnt.x += n_heavy;
                    cnt.y += n_light;
                    continue;
                }
                // this lane's place among the warp's units
                uint32_t inc = n_heavy | n_light << 16;  // at most 32 x 32 units of a step
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t v = __shfl_up_sync(full, inc, o);
                    if (lane >= o) inc += v;
                }
                const uint32_t total = __shfl_sync(full, inc, 31);
                uint32_t h = place.x + (inc & 0xffffu) - n_heavy;
                uint32_t u = nheavy * parts + place.y + (inc >> 16) - n_light;
                for (unsigned m = mask; m;) {
                    // one A tile, or all of the row's
                    const unsigned sub = pp.per_tile ? m & (0u - m) : m;
                    m &= ~sub;
                    if (n_light) {
                        units[u] = make_uint4((uint32_t)slot, (uint32_t)a0, (uint32_t)b, (uint32_t)c);
                        masks[u++] = sub;
                        continue;
                    }
                    for (uint32_t q = 0; q < parts; q++) {
                        // a heavy unit's parts: its A tiles, or quarters of them
                        // (of a single tile: quarters)
                        uint32_t x = (uint32_t)slot, pm = sub;
                        if (parts > 1) {
                            if (pp.per_tile) {
                                x |= UNIT_QUARTER | q << UNIT_QUARTER_SHIFT;
                            } else {
                                const uint32_t w = parts == 4 ? q : q >> 2;
                                // every fourth set A tile from the w-th (windows of four: one)
                                uint32_t keep = 0, n = 0;
                                for (unsigned mm = sub; mm; mm &= mm - 1u, n++)
                                    if ((n & 3u) == w) keep |= mm & (0u - mm);
                                pm = keep;
                                if (parts == 16) x |= UNIT_QUARTER | (q & 3u) << UNIT_QUARTER_SHIFT;
                            }
                        }
                        units[h * parts + q] = make_uint4(x, (uint32_t)a0, (uint32_t)b, (uint32_t)c);
                        masks[h * parts + q] = pm;
                    }
                    h++;
                }
                place.x += total & 0xffffu;
                place.y += total >> 16;
            }
        }
        if (FILL && lane == 0 && (place.x != expect.x || place.y != expect.y)) header->mismatch = 1u;
        if (!FILL) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                cnt.x += __shfl_xor_sync(full, cnt.x, o);
                cnt.y += __shfl_xor_sync(full, cnt.y, o);
            }
            if (lane == 0) row_cnt[row] = cnt;
            warp_sum.x += cnt.x;
            warp_sum.y += cnt.y;
        }
    }
    if (FILL) return;
    if (lane == 0) s_sum[warp] = warp_sum;
    if (eval) atomicAdd(&s_eval, eval);
    if (tiles) atomicAdd(&s_tiles, tiles);
    __syncthreads();
    if (threadIdx.x == 0) {
        uint2 t = make_uint2(0, 0);
        for (int w = 0; w < PLAN_WARPS; w++) {
            t.x += s_sum[w].x;
            t.y += s_sum[w].y;
        }
        block_sum[blockIdx.x] = t;
        if (s_eval) atomicAdd(&header->evaluated, s_eval);
        if (s_tiles) atomicAdd(&header->tiles, s_tiles);
    }
}

constexpr int PLAN_SCAN_THREADS = 1024;

// Exclusive scan of the block sums in place, totals at [nblocks].
__global__ void __launch_bounds__(PLAN_SCAN_THREADS)
plan_scan(uint2* block_sum, int nblocks, PlanParams pp, PlanHeader* header, uint32_t capacity) {
    __shared__ uint2 s_warp[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned long long th = 0, tl = 0;  // running totals (all threads alike)
    for (int base = 0; base < nblocks; base += PLAN_SCAN_THREADS) {
        const int i = base + (int)threadIdx.x;
        const uint2 v = i < nblocks ? block_sum[i] : make_uint2(0, 0);
        uint2 x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t a = __shfl_up_sync(0xffffffffu, x.x, o), b = __shfl_up_sync(0xffffffffu, x.y, o);
            if (lane >= o) {
                x.x += a;
                x.y += b;
            }
        }
        if (lane == 31) s_warp[warp] = x;
        __syncthreads();
        if (warp == 0) {
            uint2 w = s_warp[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t a = __shfl_up_sync(0xffffffffu, w.x, o), b = __shfl_up_sync(0xffffffffu, w.y, o);
                if (lane >= o) {
                    w.x += a;
                    w.y += b;
                }
            }
            s_warp[lane] = w;
        }
        __syncthreads();
        const uint2 before = warp ? s_warp[warp - 1] : make_uint2(0, 0), all = s_warp[31];
        if (i < nblocks) block_sum[i] = make_uint2((uint32_t)th + before.x + x.x - v.x, (uint32_t)tl + before.y + x.y - v.y);
        th += all.x;
        tl += all.y;
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        block_sum[nblocks] = make_uint2((uint32_t)th, (uint32_t)tl);
        // Few heavy units for the CTAs: cut each, so that the last ones are a
        // small share of the launch.  (DDD+DDR+DRR+RRR of 1k points: 1.50 ms
        // with whole units, 0.71 ms with sixteen units per CTA cut once,
        // 0.51 ms cut to them; 10k points have enough whole units.)
        // (single tile triples cost alike: two per CTA are enough)
        const unsigned long long want = (pp.per_tile ? 2ull : 16ull) * (unsigned)pp.slots;
        const uint32_t top = (uint32_t)pp.max_parts;
        uint32_t parts = 1;
        // (not beyond what the unit list holds)
        while (parts < top && th > 0 && th * parts < want && th * parts * 4 + tl <= capacity) parts *= 4;
        const unsigned long long n = th * parts + tl;
        header->parts = parts;
        header->needed = (uint32_t)(n < 0xffffffffull ? n : 0xffffffffull);
        header->nunits = n <= capacity ? (uint32_t)n : 0u;
    }
}

cudaError_t launch_plan(const DevJob* jobs, const uint32_t* row_off, int njobs, uint32_t nrows, const PlanParams& pp,
                        uint2* row_cnt, uint2* block_sum, PlanHeader* header, uint4* units, uint32_t* masks,
                        uint32_t capacity, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(header, 0, sizeof(PlanHeader), st);
    if (e != cudaSuccess || nrows == 0) return e;
    int rpb = 0;
    const int blocks = plan_blocks(nrows, &rpb);
    plan_rows<false><<<blocks, PLAN_WARPS * 32, 0, st>>>(jobs, row_off, njobs, nrows, rpb, pp, row_cnt, block_sum,
                                                         header, units, masks);
    plan_scan<<<1, PLAN_SCAN_THREADS, 0, st>>>(block_sum, blocks, pp, header, capacity);
    plan_rows<true><<<blocks, PLAN_WARPS * 32, 0, st>>>(jobs, row_off, njobs, nrows, rpb, pp, row_cnt, block_sum, header,
                                                        units, masks);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Triangle parametrization, guarded FP32.

// What the fast triangle kernel bins: the reference's triangle
// parametrization, JBJ, or the triangle parametrization of the double-precision
// geometry (same histogram as evaluating tp_geom for every triangle: only what
// lies in wider guard bands is).
enum FastMode : int { FAST_TP = 0, FAST_JBJ = 1, FAST_GEOM = 2 };

constexpr int TRI_WARPS = 8;
constexpr int TRI_THREADS = TRI_WARPS * 32;
constexpr int TRI_QCAP = 128;  // per-warp candidate queue: up to 63 pending + 64 new
// per j of role B: the nested sets over k of the class of side j-k (SideSet)
// and key_k >= key_j; held in shared memory as 64-entry arrays (JM_WORDS x
// TILE, word-major) so that lanes reading different j's do not share banks
constexpr int JM_WORDS = 6, JM_KEY = 5;
constexpr int SET_WORDS = 5;  // the same sets of a warp's current i
// A tiles resident at once: the tasks of a group (one job, tiles B and C
// shared) are counted up to four at a time, their points i handed out to the
// warps together
#ifndef TRI_GROUP_A_TILES
#define TRI_GROUP_A_TILES 4
#endif
constexpr int TRI_GROUP_A = TRI_GROUP_A_TILES;
// layout: tiles B, C and up to TRI_GROUP_A A tiles | j-class masks | per-warp
// i-j and i-k rows | j-k sides | per-warp candidate queues | j-k side words
// (16 bits) | histogram copies
constexpr size_t tri_tables(size_t queue_entry) {
    return (2 + TRI_GROUP_A) * TILE * sizeof(float4) +
           (JM_WORDS * TILE + TRI_WARPS * SET_WORDS) * sizeof(unsigned long long) + 2 * TRI_WARPS * TILE * sizeof(int2) +
           TILE * TILE * sizeof(float) + TRI_WARPS * TRI_QCAP * queue_entry + TILE * TILE * sizeof(short);
}
// Queue entries (14 bits) take 32 bits (10k-point estimator 13.8 ms, with 16 bits
// 14.0), but 16 for JBJ (whose four copies of 640 bins let four CTAs share an SM
// then: 5k + 5k points 14.4 ms, else 15.8) and beside the largest histograms: a
// launch has 227 KB less 1 KB for static shared memory, and up to 46,464 bins
// must fit.
constexpr int TRI_WIDE_QUEUE_BINS = 46256;
constexpr bool tri_wide_queue(int hist_len, bool jbj) { return !jbj && hist_len <= TRI_WIDE_QUEUE_BINS; }
constexpr size_t TRI_SMEM_WIDE = tri_tables(sizeof(uint32_t)), TRI_SMEM_NARROW = 45568;
static_assert(TRI_SMEM_WIDE + 4 * TRI_WIDE_QUEUE_BINS <= 226 * 1024 && TRI_SMEM_NARROW + 4 * 46464 <= 226 * 1024 &&
              tri_tables(sizeof(uint16_t)) <= TRI_SMEM_NARROW, "fast triangle layout");
// (the plain FP64 kernel's layout -- three tiles, a j-k table of int2 and one
// row per warp -- fits the same allocation)
static_assert(TRI_SMEM_NARROW >= 3 * TILE * sizeof(float4) + TILE * TILE * sizeof(int2) + TRI_WARPS * TILE * sizeof(int2),
              "FP64 triangle layout");

// Side word of the fast kernel: code16 * 128 + class weight, 16 bits (see
// engine.h); code16 is the s-bin itself.
// (A division-free s-bin -- a guess corrected against exact thresholds
// staged in shared memory -- measured slower: 14.19 vs 13.95 ms on the
// default workload.)
template <int MODE>
__device__ __forceinline__ int tri_side_word(float d, const TriParams& p) {
    int code, w;
    if (MODE == FAST_GEOM) {
        // a side whose double length may fall on the other side of s_lo or
        // s_hi counts as in range (the class that rejects least); the guard
        // band of its s coordinate sends its triangles to the recheck.  A zero
        // side is no reason to reject: its double length may not be zero.
        if (d < p.geo_s_below) return CODE16_BELOW * 128 + (d >= p.lmax ? CW_REJECT : CW_BELOW);
        if (d >= p.geo_s_above) return CODE16_ABOVE * 128 + (d >= p.lmax ? CW_REJECT : CW_ABOVE);
        code = __float2int_rz(__fdiv_rn(__fsub_rn(d, p.s_lo), p.s_bw));
        return min(max(code, 0), p.S - 1) * 128 + CW_IN;
    }
    if (d == 0.f) {
        code = CODE16_ZERO;
        w = CW_REJECT;
    } else if (d < p.s_lo) {
        code = CODE16_BELOW;
        w = CW_BELOW;
    } else if (d >= p.s_hi) {
        code = CODE16_ABOVE;
        w = CW_ABOVE;
    } else {
        code = __float2int_rz(__fdiv_rn(__fsub_rn(d, p.s_lo), p.s_bw));
        w = code < p.S ? CW_IN : CW_ABOVE;  // code == S: rounding at the top edge, index past the array
    }
    if (d >= p.lmax) w = CW_REJECT;
    return code * 128 + w;
}

// 1.5 * 2^23: adding it rounds a float in (-2^22, 2^22) to an integer held in
// the low mantissa bits.
#define MAGIC 12582912.0f
#define MAGIC_BITS 0x4B400000

struct GuardedBin {
    int bin;      // floor of the bin coordinate (valid if not near an edge)
    float err;    // signed distance of the coordinate from its bin centre (in [-0.5, 0.5])
};

// f_m = coordinate - 0.5; returns floor(coordinate) and the offset used by the guard
__device__ __forceinline__ GuardedBin magic_floor(float f_m) {
    float tm = __fadd_rn(f_m, MAGIC);
    float dd = __fsub_rn(tm, MAGIC);
    GuardedBin g;
    g.bin = __float_as_int(tm) - MAGIC_BITS;
    g.err = __fsub_rn(f_m, dd);
    return g;
}

__device__ __forceinline__ unsigned weight_index(int wa, int wb, int wc) { return (unsigned)(wa + wb + wc) & 127u; }
__device__ __forceinline__ bool mask_bit(unsigned mask, unsigned idx) { return (__funnelshift_rc(mask, 0u, idx) & 1u) != 0; }

// Two floats in one 64-bit register for the packed FP32 instructions of
// sm_100+ (add/sub/mul/fma .rn .f32x2: two IEEE single operations per
// instruction, each element rounded exactly as the scalar operation).  Unlike
// the scalar __fmul_rn/__fadd_rn intrinsics, a packed product that feeds a
// packed sum is contracted into one fma.f32x2 by ptxas (measured: the packed
// squared side sums differ from the scalar ones in a fifth of the cases), so
// only results whose exact rounding does not matter, or that no contraction
// can reach, are computed packed.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pk2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void up2(f32x2 r, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(r)); }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f32x2 splat2(float a) { return pk2(a, a); }

// magic_floor of two coordinates
__device__ __forceinline__ void magic_floor2(f32x2 f_m, int& b0, int& b1, float& e0, float& e1) {
    const f32x2 mg = splat2(MAGIC);
    const f32x2 tm = add2(f_m, mg);
    up2(sub2(f_m, sub2(tm, mg)), e0, e1);
    float t0, t1;
    up2(tm, t0, t1);
    b0 = __float_as_int(t0) - MAGIC_BITS;
    b1 = __float_as_int(t1) - MAGIC_BITS;
}

// The same with the bins left as the bits of coordinate + MAGIC: compared
// against MAGIC_BITS + n, and with the offset folded into an address base.
__device__ __forceinline__ void magic_bits2(f32x2 f_m, uint32_t& b0, uint32_t& b1, float& e0, float& e1) {
    const f32x2 mg = splat2(MAGIC);
    const f32x2 tm = add2(f_m, mg);
    up2(sub2(f_m, sub2(tm, mg)), e0, e1);
    float t0, t1;
    up2(tm, t0, t1);
    b0 = __float_as_uint(t0);
    b1 = __float_as_uint(t1);
}

// Counts one at a 32-bit shared-memory address (address arithmetic modulo
// 2^32, so that a base may hold the MAGIC_BITS offset of a bin).  Barriers
// order it with the flush's plain reads, as they do atomicAdd.  What is not
// counted goes to a word that nobody reads: lanes that hit one address cost one
// access, a branch around each atomic costs three instructions (pairs of 50k
// points: 24 -> 18 instructions a pair).
__device__ __forceinline__ uint32_t shared_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void count_at(uint32_t addr) { asm volatile("red.shared.add.u32 [%0], 1;" ::"r"(addr)); }
// A predicated 16-bit store to a 32-bit shared-memory address (no branch).
__device__ __forceinline__ void store_if(bool ok, uint32_t addr, uint32_t v) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p st.shared.u16 [%0], %1;\n\t}" ::"r"(addr),
                 "h"((unsigned short)v), "r"((unsigned)ok)
                 : "memory");
}
// UNIT: every weight is one
template <bool UNIT>
__device__ __forceinline__ void count_at(uint32_t addr, unsigned w) {
    if (UNIT) count_at(addr);
    else asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(addr), "r"(w));
}

// theta_fast of two cosines; t: 1 - |c|, y: its reciprocal square root
__device__ __forceinline__ void theta_fast2(f32x2 c, const TriParams& p, f32x2& f_m, f32x2& thr, f32x2& t, f32x2& y) {
    float c0, c1;
    up2(c, c0, c1);
    const f32x2 x = pk2(fabsf(c0), fabsf(c1));
    t = sub2(splat2(1.0f), x);
    float t0, t1;
    up2(t, t0, t1);
    y = pk2(rsqrt_approx(t0), rsqrt_approx(t1));
    const f32x2 sq = mul2(t, y);
    f32x2 P = splat2(p.t_coef[5]);
    P = fma2(P, x, splat2(p.t_coef[4]));
    P = fma2(P, x, splat2(p.t_coef[3]));
    P = fma2(P, x, splat2(p.t_coef[2]));
    P = fma2(P, x, splat2(p.t_coef[1]));
    P = fma2(P, x, splat2(p.t_coef[0]));
    float a0, a1;
    up2(fma2(sq, P, splat2(-p.t_half)), a0, a1);  // K*acos(|c|) - K*pi/2
    a0 = __int_as_float(__float_as_int(a0) ^ (__float_as_int(c0) & 0x80000000));  // acos(-x) = pi - acos(x)
    a1 = __int_as_float(__float_as_int(a1) ^ (__float_as_int(c1) & 0x80000000));
    f_m = add2(pk2(a0, a1), splat2(p.t_off0));
    thr = fma2(splat2(-p.t_thrB), y, splat2(p.t_thrA));
}

// Full fast path of two triangles at once (each lane's two candidates): sides
// a, b, c with their words; w: multiplicities (0 = none).  The FP32
// arithmetic of the two runs in packed f32x2 instructions.  A triangle whose
// weight index says some permutation may count is binned into Hw, unless a
// permutation that could count has a coordinate inside its guard band: then
// guard[t] is set and the triangle must be recomputed exactly.
//
// GEOM: the double-precision geometry is approximated instead of the
// reference's floats.  With u = 2^-24 a float side is within 3.5 u of its double
// length, so a ratio is within 11 u (twice that where two sides within rounding
// change places), and a cosine within 4e-6 E, E = (s^2 + m^2 + l^2) / (2 s m) the
// amplification of its cancelling numerator (12 u E for the sides and
// roundings, doubled for changed places, and a margin).  An angle moves by at
// most 1.42 dc / sqrt(1 - |c|), and a cosine within 2 dc of +-1 is always
// recomputed.  (Every triangle in double is bound by the FP64 pipe, two lanes a
// clock and SM: DDD+DDR+DRR+RRR of 1k points 251 ms; so 0.65 ms, 0.2 % of the
// binned triangles recomputed.)
template <bool THETA_FULL, bool GEOM, bool UNIT>
__device__ __forceinline__ void triangle_full2(const float (&a)[2], const int (&wa)[2], const float (&b)[2],
                                               const int (&wb)[2], const float (&c)[2], const int (&wc)[2],
                                               const unsigned (&w)[2], const TriParams& p, unsigned int* Hw,
                                               unsigned int* dump, bool (&guard)[2]) {
    float s[2], m[2], l[2];
    int off_s[2], off_m[2];
    bool v02[2], v1[2];
#pragma unroll
    for (int t = 0; t < 2; t++) {
        const unsigned idx = weight_index(wa[t], wb[t], wc[t]);
        v02[t] = w[t] && mask_bit(VALID_02, idx);
        v1[t] = w[t] && mask_bit(VALID_1, idx);
        const float lo_ab = fminf(a[t], b[t]), hi_ab = fmaxf(a[t], b[t]);
        s[t] = fminf(lo_ab, c[t]);
        l[t] = fmaxf(hi_ab, c[t]);
        m[t] = fmaxf(lo_ab, fminf(hi_ab, c[t]));
        const int wlo = min(wa[t], wb[t]), whi = max(wa[t], wb[t]);
        // s-bins of the shortest and the middle side, times Q
        off_s[t] = (min(wlo, wc[t]) >> 7) * p.Q;
        off_m[t] = (max(wlo, min(whi, wc[t])) >> 7) * p.Q;
    }
    const f32x2 S = pk2(s[0], s[1]), M = pk2(m[0], m[1]), L = pk2(l[0], l[1]);
    // the squares enter the cosine numerators as the reference rounds them:
    // scalar products (ptxas contracts a packed mul.rn.f32x2 feeding an
    // add.rn.f32x2 into fma.f32x2, measured on sm_103a, which would change
    // the numerators' rounding)
    const f32x2 S2 = pk2(__fmul_rn(s[0], s[0]), __fmul_rn(s[1], s[1]));
    const f32x2 M2 = pk2(__fmul_rn(m[0], m[0]), __fmul_rn(m[1], m[1]));
    const f32x2 L2 = pk2(__fmul_rn(l[0], l[0]), __fmul_rn(l[1], l[1]));
    const f32x2 qs = splat2(p.q_scale), qo = splat2(p.q_off);
    const f32x2 rsq = mul2(pk2(rcp_approx(s[0]), rcp_approx(s[1])), qs);
    const f32x2 rmq = mul2(pk2(rcp_approx(m[0]), rcp_approx(m[1])), qs);
    int q0b[2], q1b[2], q2b[2], t0b[2], t1b[2], t2b[2];
    float q0e[2], q1e[2], q2e[2], t0e[2], t1e[2], t2e[2];
    magic_floor2(fma2(M, rsq, qo), q0b[0], q0b[1], q0e[0], q0e[1]);
    magic_floor2(fma2(L, rmq, qo), q1b[0], q1b[1], q1e[0], q1e[1]);
    magic_floor2(fma2(L, rsq, qo), q2b[0], q2b[1], q2e[0], q2e[1]);
    const f32x2 num0 = sub2(add2(S2, M2), L2);
    const f32x2 num1 = sub2(add2(M2, L2), S2);
    float sm0, sm1, ml0, ml1;
    up2(mul2(S, M), sm0, sm1);
    up2(mul2(M, L), ml0, ml1);
    const f32x2 half = splat2(0.5f);
    const f32x2 c0 = mul2(mul2(num0, pk2(rcp_approx(sm0), rcp_approx(sm1))), half);
    const f32x2 c1 = mul2(mul2(num1, pk2(rcp_approx(ml0), rcp_approx(ml1))), half);
    f32x2 f0m, thr0, f1m, thr1, tc0, tc1, y0, y1;
    theta_fast2(c0, p, f0m, thr0, tc0, y0);
    theta_fast2(c1, p, f1m, thr1, tc1, y1);
    bool gs[2] = {false, false}, gm[2] = {false, false};
    if (GEOM) {
        const f32x2 sum2 = add2(add2(S2, M2), L2);
        const f32x2 E0 = mul2(mul2(sum2, pk2(rcp_approx(sm0), rcp_approx(sm1))), half);
        const f32x2 E1 = mul2(mul2(sum2, pk2(rcp_approx(ml0), rcp_approx(ml1))), half);
        float e0[2], e1[2], t0[2], t1[2], h0[2], h1[2], x0[2], x1[2], sv[2], mv[2];
        up2(E0, e0[0], e0[1]);
        up2(E1, e1[0], e1[1]);
        up2(tc0, t0[0], t0[1]);
        up2(tc1, t1[0], t1[1]);
        up2(fma2(splat2(-p.geo_t), mul2(E0, y0), splat2(p.t_thrA)), h0[0], h0[1]);
        up2(fma2(splat2(-p.geo_t), mul2(E1, y1), splat2(p.t_thrA)), h1[0], h1[1]);
        int b0, b1;
        magic_floor2(fma2(S, splat2(p.geo_s_inv), splat2(p.geo_s_off)), b0, b1, sv[0], sv[1]);
        magic_floor2(fma2(M, splat2(p.geo_s_inv), splat2(p.geo_s_off)), b0, b1, mv[0], mv[1]);
#pragma unroll
        for (int t = 0; t < 2; t++) {
            x0[t] = t0[t] > 8e-6f * e0[t] ? h0[t] : -1.f;
            x1[t] = t1[t] > 8e-6f * e1[t] ? h1[t] : -1.f;
            gs[t] = !(fabsf(sv[t]) <= p.geo_s_thr);
            gm[t] = !(fabsf(mv[t]) <= p.geo_s_thr);
        }
        thr0 = pk2(x0[0], x0[1]);
        thr1 = pk2(x1[0], x1[1]);
    }
    const f32x2 f2m = sub2(sub2(splat2(p.t2_off), f0m), f1m);
    float thr0v[2], thr1v[2], thr2v[2];
    up2(thr0, thr0v[0], thr0v[1]);
    up2(thr1, thr1v[0], thr1v[1]);
    up2(add2(add2(thr0, thr1), splat2(-0.5f - 1e-6f)), thr2v[0], thr2v[1]);
    magic_floor2(f0m, t0b[0], t0b[1], t0e[0], t0e[1]);
    magic_floor2(f1m, t1b[0], t1b[1], t1e[0], t1e[1]);
    magic_floor2(f2m, t2b[0], t2b[1], t2e[0], t2e[1]);
#pragma unroll
    for (int t = 0; t < 2; t++) {
        // guard: a permutation that could count has a value near a bin edge
        const bool gq0 = !(fabsf(q0e[t]) <= p.q_thr), gq1 = !(fabsf(q1e[t]) <= p.q_thr),
                   gq2 = !(fabsf(q2e[t]) <= p.q_thr);
        const bool gt0 = !(fabsf(t0e[t]) <= thr0v[t]), gt1 = !(fabsf(t1e[t]) <= thr1v[t]),
                   gt2 = !(fabsf(t2e[t]) <= thr2v[t]);
        const bool g = (v02[t] && (gq0 || gt0 || gq2 || gt2 || gs[t])) || (v1[t] && (gq1 || gt1 || gm[t]));
        bool ok0 = v02[t] && !g && (unsigned)q0b[t] < (unsigned)p.Q;
        bool ok1 = v1[t] && !g && (unsigned)q1b[t] < (unsigned)p.Q;
        bool ok2 = v02[t] && !g && (unsigned)q2b[t] < (unsigned)p.Q;
        if (!THETA_FULL) {
            ok0 = ok0 && (unsigned)t0b[t] < (unsigned)p.T;
            ok1 = ok1 && (unsigned)t1b[t] < (unsigned)p.T;
            ok2 = ok2 && (unsigned)t2b[t] < (unsigned)p.T;
        }
        // (uncounted permutations add to the lane's dump word: no branches)
        const uint32_t base = shared_addr(Hw), none = shared_addr(dump);
        count_at<UNIT>(ok0 ? base + 4u * (uint32_t)((off_s[t] + q0b[t]) * p.T + t0b[t]) : none, w[t]);
        count_at<UNIT>(ok1 ? base + 4u * (uint32_t)((off_m[t] + q1b[t]) * p.T + t1b[t]) : none, w[t]);
        count_at<UNIT>(ok2 ? base + 4u * (uint32_t)((off_s[t] + q2b[t]) * p.T + t2b[t]) : none, w[t]);
        guard[t] = g;
    }
}

// JBJ binning of two triangles (src/3pcf_C_version_triangle_parametrization_JBJ.cc
// distance(), :116-229): one permutation, s = shortest, q = s/m and
// theta = (l - m)/s in float, binned as distance_to_bin does.  The coordinates
// come from rcp.approx in packed instructions; one inside the guard band of a
// bin edge (1e-6 of the coordinate range: the reciprocal's two ulps and the
// roundings of either side are below 6e-7 of it) is recomputed with the
// reference's own divisions.  The s-bin comes from the shortest side's word; a
// triangle whose weight index says its shortest side is out of range, zero or
// rejected, or whose multiplicity is 0, adds nothing.  (Four IEEE divisions for
// every triangle: 20.6 ms instead of 18.5 on 5k + 5k points.)

// distance_to_bin: -1 outside [lo, hi); the bin as the reference truncates it,
// which rounding can make n at the top edge (the index then runs into the
// next row, as the reference's does, or past the array)
__device__ __forceinline__ int jbj_axis_bin(float v, float lo, float hi, float bw) {
    if (!(v >= lo) || v >= hi) return -1;  // (v is never NaN here: no zero side reaches this)
    return __float2int_rz(__fdiv_rn(__fsub_rn(v, lo), bw));
}

template <bool UNIT>
__device__ __forceinline__ void jbj_full2(const float (&a)[2], const int (&wa)[2], const float (&b)[2],
                                          const int (&wb)[2], const float (&c)[2], const int (&wc)[2],
                                          const unsigned (&w)[2], const TriParams& p, unsigned int* Hw,
                                          unsigned int* dump) {
    float s[2], m[2], l[2];
    int code[2];
    bool v[2];
#pragma unroll
    for (int t = 0; t < 2; t++) {
        v[t] = w[t] && mask_bit(VALID_02, weight_index(wa[t], wb[t], wc[t]));
        const float lo_ab = fminf(a[t], b[t]), hi_ab = fmaxf(a[t], b[t]);
        s[t] = fminf(lo_ab, c[t]);
        l[t] = fmaxf(hi_ab, c[t]);
        m[t] = fmaxf(lo_ab, fminf(hi_ab, c[t]));
        code[t] = min(min(wa[t], wb[t]), wc[t]) >> 7;  // s-bin of the shortest side
    }
    const f32x2 S = pk2(s[0], s[1]), M = pk2(m[0], m[1]), L = pk2(l[0], l[1]);
    const f32x2 q = mul2(S, pk2(rcp_approx(m[0]), rcp_approx(m[1])));
    const f32x2 th = mul2(sub2(L, M), pk2(rcp_approx(s[0]), rcp_approx(s[1])));
    int i1[2], i2[2];
    float e1[2], e2[2];
    magic_floor2(fma2(q, splat2(p.q_scale), splat2(p.q_off)), i1[0], i1[1], e1[0], e1[1]);
    magic_floor2(fma2(th, splat2(p.t_coef[0]), splat2(p.t_off0)), i2[0], i2[1], e2[0], e2[1]);
    const uint32_t base = shared_addr(Hw), none = shared_addr(dump);
#pragma unroll
    for (int t = 0; t < 2; t++) {
        const bool safe = fabsf(e1[t]) <= p.q_thr && fabsf(e2[t]) <= p.t_thrA;
        const bool take = v[t] && safe && (unsigned)i1[t] < (unsigned)p.Q && (unsigned)i2[t] < (unsigned)p.T;
        count_at<UNIT>(take ? base + 4u * (uint32_t)((code[t] * p.Q + i1[t]) * p.T + i2[t]) : none, w[t]);
        if (v[t] && !safe) {
            const int x1 = jbj_axis_bin(__fdiv_rn(s[t], m[t]), p.q_lo, p.q_hi, p.q_bw);
            const int x2 = jbj_axis_bin(__fdiv_rn(__fsub_rn(l[t], m[t]), s[t]), p.t_lo, p.t_hi, p.t_bw);
            const int x = (code[t] * p.Q + x1) * p.T + x2;
            if (x1 >= 0 && x2 >= 0 && x < p.len) atomicAdd(Hw + x, w[t]);
        }
    }
}

__device__ __forceinline__ void push_recheck(const RecheckQueue& q, uint32_t slot, unsigned w, uint32_t ia, uint32_t ib,
                                             uint32_t ic) {
    unsigned int pos = atomicAdd(q.count, 1u);
    if (pos < q.cap) q.items[pos] = make_uint4(slot | (w << RECHECK_WEIGHT_SHIFT), ia, ib, ic);
}

struct TaskGeom {
    int a0, nA, b0, nB, c0, nC;
};

__device__ __forceinline__ TaskGeom task_geom(const DevJob& J, uint4 task) {
    TaskGeom g;
    g.a0 = J.tile_start[0][task.y];
    g.nA = J.tile_start[0][task.y + 1] - g.a0;
    g.b0 = J.tile_start[1][task.z];
    g.nB = J.tile_start[1][task.z + 1] - g.b0;
    g.c0 = J.tile_start[2][task.w];
    g.nC = J.tile_start[2][task.w + 1] - g.c0;
    return g;
}

__device__ __forceinline__ void load_points(float4* P, const DevJob& J, const TaskGeom& g) {
    for (int t = threadIdx.x; t < 3 * TILE; t += blockDim.x) {
        int role = t / TILE, idx = t % TILE;
        int n = role == 0 ? g.nA : (role == 1 ? g.nB : g.nC);
        int base = role == 0 ? g.a0 : (role == 1 ? g.b0 : g.c0);
        P[t] = idx < n ? J.pts[role][base + idx] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
}

__device__ __forceinline__ int pkey(float4 p) { return __float_as_int(p.w); }

// What a unit's CTA shares beside the tiles: boxes (lo, hi) of tiles B and C
// and of all A tiles of the unit, and the resident A tiles (first point,
// points, TRI_* flags, position of the first point in its tile).
// floats as ints of the same order (its own inverse)
__device__ __forceinline__ int ordered_int(float x) {
    const int v = __float_as_int(x);
    return v ^ ((v >> 31) & 0x7fffffff);
}
__device__ __forceinline__ float ordered_float(int v) { return __int_as_float(v ^ ((v >> 31) & 0x7fffffff)); }

// Extends a box in shared memory by those of the warp's lanes that have one.
__device__ __forceinline__ void box_add(int* box, int lane, bool has, float4 lo, float4 hi) {
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const float l = a == 0 ? lo.x : (a == 1 ? lo.y : lo.z), h = a == 0 ? hi.x : (a == 1 ? hi.y : hi.z);
        const int mn = __reduce_min_sync(0xffffffffu, has ? ordered_int(l) : INT_MAX);
        const int mx = __reduce_max_sync(0xffffffffu, has ? ordered_int(h) : INT_MIN);
        if (lane == 0) {
            atomicMin(box + a, mn);
            atomicMax(box + 3 + a, mx);
        }
    }
}

struct TriShared {
    uint4 unit;
    uint32_t mask;
    uint32_t pred;       // loop nest of the unit's job
    int b0, c0;          // first points of tiles B and C
    int next_i, end_i;  // points listed of the resident A tiles: handed out, and their number
    uint8_t list[TRI_GROUP_A * TILE];
    float box[2][6];
    int abox[6];         // box of the unit's listed points (of its A tiles, if they are not all resident), ordered_int
    int nj, nk;          // points of tiles B and C listed: their number and their places in the tiles, ascending
    uint8_t jlist[TILE], klist[TILE];
    int4 meta[TRI_GROUP_A];
    unsigned int dump[32];  // counts of permutations that do not count, by lane
};
static_assert(TRI_GROUP_A * TILE <= 256 && TRI_GROUP_A * TILE <= TRI_THREADS, "one thread and one byte per listed point");

// Queued candidate triangle of the current i: j (bits 0-5), k (bits 6-11) and
// its weight (bits 12-13).

// Runs the full binning path on n (<= 64) queued candidates, two per lane
// (packed into the f32x2 instructions of one binning path).
template <bool THETA_FULL, int MODE, bool UNIT, typename Entry>
__device__ __forceinline__ void run_candidates(const Entry* cand, int n, const int2* row_ij, const int2* row_ik,
                                               const float* JKd, const short* JKw, const TriParams& p, unsigned int* Hw,
                                               RecheckQueue& q, TriShared& S, uint32_t ia) {
    const int lane = threadIdx.x & 31;
    const uint32_t e0 = lane < n ? cand[lane] : 0u;
    const uint32_t e1 = lane + 32 < n ? cand[lane + 32] : 0u;
    const int j0 = e0 & 63, k0 = (e0 >> 6) & 63, j1 = e1 & 63, k1 = (e1 >> 6) & 63;
    const unsigned w0 = e0 >> 12, w1 = e1 >> 12;
    const int2 ij0 = row_ij[j0], ik0 = row_ik[k0];
    const int2 ij1 = row_ij[j1], ik1 = row_ik[k1];
    const float fa[2] = {__int_as_float(ij0.x), __int_as_float(ij1.x)};
    const float fb[2] = {__int_as_float(ik0.x), __int_as_float(ik1.x)};
    const float fc[2] = {JKd[j0 * TILE + k0], JKd[j1 * TILE + k1]};
    const int wa[2] = {ij0.y, ij1.y}, wb[2] = {ik0.y, ik1.y};
    const int wc[2] = {JKw[j0 * TILE + k0], JKw[j1 * TILE + k1]};
    const unsigned ww[2] = {w0, w1};
    if (MODE == FAST_JBJ) {
        jbj_full2<UNIT>(fa, wa, fb, wb, fc, wc, ww, p, Hw, S.dump + lane);
        return;
    }
    bool guard[2];
    triangle_full2<THETA_FULL, MODE == FAST_GEOM, UNIT>(fa, wa, fb, wb, fc, wc, ww, p, Hw, S.dump + lane, guard);
    const bool g0 = guard[0], g1 = guard[1];
    const uint32_t slot = S.unit.x & UNIT_SLOT_MASK;
    if (g0) push_recheck(q, slot, w0, ia, (uint32_t)(S.b0 + S.jlist[j0]), (uint32_t)(S.c0 + S.klist[k0]));
    if (g1) push_recheck(q, slot, w1, ia, (uint32_t)(S.b0 + S.jlist[j1]), (uint32_t)(S.c0 + S.klist[k1]));
}

// Side classes for candidate filtering: none (zero length or too long), X below
// s_lo or from q_hi s_hi up, M2 and M1 from q_hi s_split and from s_hi up, I1 and
// I2 the s range below and from s_split.  Their sets are nested by the order of
// the numbers: all, Q without X, R without M2, I the s range, I2.
//
// A counted triangle has two sides one of which is an I and the other the next
// longer one within q_hi of it (permutation 0/2: the shortest and the middle
// one; permutation 1: the middle and the longest).  So its classes hold one of
// the pairs I-I, I1-M1, I2-M1, I2-M2, whatever the third side is.  JBJ is
// permutation 0 with 1/q_lo for q_hi.
enum SideClass : int { SC_NONE = 0, SC_X = 1, SC_M2 = 2, SC_M1 = 3, SC_I1 = 4, SC_I2 = 5 };
enum SideSet : int { SET_ALL = 0, SET_Q = 1, SET_R = 2, SET_I = 3, SET_I2 = 4 };  // class > number

template <int MODE>
__device__ __forceinline__ int side_class(int word, float d, const TriParams& p) {
    const int w = word & 127;
    if (w >= CW_REJECT) return SC_NONE;
    if (w == CW_BELOW) return MODE == FAST_JBJ ? SC_NONE : SC_X;  // (JBJ counts no triangle with such a side)
    if (w == CW_IN) return d < p.s_split ? SC_I1 : SC_I2;
    return d < p.mid_split ? SC_M1 : d < p.mid_hi ? SC_M2 : SC_X;
}

__device__ __forceinline__ unsigned long long ballot64(bool lo, bool hi) {
    return (unsigned long long)__ballot_sync(0xffffffffu, lo) | ((unsigned long long)__ballot_sync(0xffffffffu, hi) << 32);
}

// The nested sets of the sides of one point, lane and lane + 32, written by one
// lane at the given stride.
__device__ __forceinline__ unsigned long long side_sets(unsigned long long* out, int stride, int lane, int c0, int c1) {
    const unsigned long long all = ballot64(c0 > SET_ALL, c1 > SET_ALL), q = ballot64(c0 > SET_Q, c1 > SET_Q),
                             r = ballot64(c0 > SET_R, c1 > SET_R), i = ballot64(c0 > SET_I, c1 > SET_I),
                             i2 = ballot64(c0 > SET_I2, c1 > SET_I2);
    if (lane == 0) {
        out[SET_ALL * stride] = all;
        out[SET_Q * stride] = q;
        out[SET_R * stride] = r;
        out[SET_I * stride] = i;
        out[SET_I2 * stride] = i2;
    }
    return all;
}

// Candidate k's of a pair (i, j) whose side i-j has class cij, from the sets of
// the sides i-k (n) and j-k (m, at stride TILE): a class that makes a pair with
// cij, or one of the pairs between i-k and j-k (exactly those beside M2; beside
// X also I1-M2, beside an I or M1 they are in the first kind).  (With one class I
// and one M 22 % more triangles of the 10k-point estimator reach the binning:
// kernel 9.7 ms, so 8.7; without I2's set 12 % more and 9.5.)
__device__ __forceinline__ unsigned long long candidate_mask(int cij, const unsigned long long* n, const unsigned long long* m) {
    const int with = cij == SC_X ? SET_Q : SET_R;
    unsigned long long cm = (n[SET_I] & m[with * TILE]) | (n[with] & m[SET_I * TILE]);
    const int pairs = SC_M2 + SET_I2 - cij;  // the set of the classes that make a pair with cij (but X)
    if (cij != SC_X) cm |= n[SET_ALL] & m[SET_ALL * TILE] & (n[pairs] | m[pairs * TILE]);
    return cm;
}
static_assert(SC_M1 + SET_I == SC_M2 + SET_I2 && SC_I1 + SET_R == SC_M2 + SET_I2 && SC_I2 + SET_Q == SC_M2 + SET_I2,
              "classes and the sets of those that make a pair with them");

// (UNIT: loop nests without or with a 0/1 weight; else those of two arrays.  The
// nest itself is a value, not a template argument: five copies of the code cost
// batches of unlike jobs, whose CTAs run different nests at a time, a fifth: 100
// voxels 2.34 -> 1.92 ms, most of it by the second place that bins, DDD+DDR+DRR+
// RRR of 1k points 0.465 -> 0.442.  One copy for both costs the weights of all
// and more registers: 10k-point estimator 9.9 -> 10.5.)
template <bool UNIT, bool THETA_FULL, int MODE, typename Entry>
__device__ void triangle_group_fast(const DevJob* __restrict__ jobs, const TriParams& p, float4* P, float* JKd, short* JKw, int2* IJ,
                                    int2* IK, Entry* Q, unsigned long long* JM, TriShared& S, unsigned int* Hw,
                                    RecheckQueue& q, unsigned long long& evaluated, unsigned long long& binned) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float4 *PB = P, *PC = P + TILE, *PA = P + 2 * TILE;
    // every triple of the unit has the same job and tiles B and C
    bool diag_jk;
    int numB, numC;  // points of B and C (that can count, once these are listed)
    {
        const DevJob& J = jobs[S.unit.x & UNIT_SLOT_MASK];
        diag_jk = (J.mode & JOB_C_FROM_B) && S.unit.z == S.unit.w;
        numB = J.tile_start[1][S.unit.z + 1] - J.tile_start[1][S.unit.z];
        numC = J.tile_start[2][S.unit.w + 1] - J.tile_start[2][S.unit.w];
    }
    // a side that provably reaches lmax is rejected whatever its exact value:
    // points farther than that from a whole tile take no part in the task
    // (the 1e-5 margin covers the rounding of the bound and of the distance)
    const float reach = p.lmax * (1.0f + 1e-5f);
    const float reach2 = reach * reach;
    bool have_jk = false;  // the j-k sides are in the tables
    int2* row_ij = IJ + warp * TILE;
    int2* row_ik = IK + warp * TILE;
    Entry* cand = Q + warp * TRI_QCAP;
    unsigned long long* sets = JM + JM_WORDS * TILE + warp * SET_WORDS;
    int key_k0 = 0, key_k1 = 0;
    unsigned ev = 0, bn = 0;
    // A tiles of the unit, up to TRI_GROUP_A at a time
    for (int ch = 0; ch < __popc(S.mask); ch += TRI_GROUP_A) {
        // (read again for every chunk: no registers held across the i loop)
        const uint4 unit = S.unit;
        const DevJob& J = jobs[unit.x & UNIT_SLOT_MASK];
        const int tb0 = J.tile_start[1][unit.z], tc0 = J.tile_start[2][unit.w];
        const int nr = min(TRI_GROUP_A, __popc(S.mask) - ch);
        // points of each A tile the unit covers: all, or a quarter
        const int ifrom = unit.x & UNIT_QUARTER ? (int)((unit.x >> UNIT_QUARTER_SHIFT) & 3u) * (TILE / 4) : 0;
        const int ilen = unit.x & UNIT_QUARTER ? TILE / 4 : TILE;
        auto tile_of = [&](int r) {  // the (ch + r)-th A tile of the mask
            uint32_t m = S.mask;
            for (int x = 0; x < ch + r; x++) m &= m - 1u;
            return (int)unit.y + __ffs(m) - 1;
        };
        if (ch > 0) __syncthreads();  // the previous tiles' i loops are done
        // tiles B and C (once) and the A tiles, tile r at PA + r * TILE
        for (int tt = (ch == 0 ? 0 : 2 * TILE) + threadIdx.x; tt < (2 + nr) * TILE; tt += blockDim.x) {
            const int idx = tt % TILE;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (tt < TILE) {
                if (idx < numB) v = J.pts[1][tb0 + idx];
            } else if (tt < 2 * TILE) {
                if (idx < numC) v = J.pts[2][tc0 + idx];
            } else {
                const int a = tile_of(tt / TILE - 2), a0 = J.tile_start[0][a] + ifrom;
                if (idx < ilen && a0 + idx < J.tile_start[0][a + 1]) v = J.pts[0][a0 + idx];
            }
            P[tt] = v;
        }
        if (threadIdx.x < nr) {
            const int a = tile_of(threadIdx.x), a0 = J.tile_start[0][a];
            const int n = min(ilen, J.tile_start[0][a + 1] - a0 - ifrom);
            // first point, points (of the quarter), which j come after point i: those from i + w + 1, or all
            S.meta[threadIdx.x] = make_int4(a0 + ifrom, n, (J.mode & JOB_B_FROM_A) && a == (int)unit.z, ifrom);
        }
        if (ch == 0 && warp == 1) {  // boxes of tiles B and C
            if (lane < 12) {
                const int role = lane < 6 ? 1 : 2, f = lane % 6;
                const float4 v = J.box[role][2 * (size_t)(role == 1 ? unit.z : unit.w) + f / 3];
                S.box[role - 1][f] = f % 3 == 0 ? v.x : (f % 3 == 1 ? v.y : v.z);
            }
        }
        if (threadIdx.x == 0) {
            S.next_i = 0;
            S.end_i = 0;
            S.b0 = tb0;
            S.c0 = tc0;
        }
        if (ch == 0 && threadIdx.x < 6) S.abox[threadIdx.x] = threadIdx.x < 3 ? INT_MAX : INT_MIN;
        __syncthreads();
        // The points that may be part of a counted triangle, listed by one
        // thread each: by the lower bounds of its sides, all below lmax, one in
        // the s range and another below mid_hi.  (Handed out untested, 56 % of
        // the points of the 10k-point estimator and 77 % of those of 100 voxels
        // cost a warp a draw and a test of its own to be dropped, and others a
        // scan of the j by which no candidate came: kernels 11.4 -> 10.0 ms and
        // 3.42 -> 2.56 ms.)  A point that is not a number lies outside its
        // tile's box, and a side with it is in the s range: with such points
        // only i out of reach of a whole tile are left out.
        auto possible = [&](float x2, float y2, float z2) {
            const float lo = fminf(x2, y2), hi = fmaxf(x2, y2), in = p.s_hi * (1.0f + 1e-5f), next = p.mid_hi * (1.0f + 1e-5f);
            // (an infinite limit keeps an infinite distance too)
            return !(fminf(lo, z2) > in * in) && !(fmaxf(lo, fminf(hi, z2)) > next * next) && !(fmaxf(hi, z2) > reach2);
        };
        // squared distances of a point from two boxes and of these from one another
        auto bounds2 = [&](float4 pt, auto b_lo, auto b_hi, const float* c, float& pb, float& pc, float& bc) {
            pb = pc = bc = 0.f;
#pragma unroll
            for (int a = 0; a < 3; a++) {
                const float v = a == 0 ? pt.x : (a == 1 ? pt.y : pt.z);
                const float bl = b_lo(a), bh = b_hi(a), cl = c[a], ch = c[3 + a];
                const float gb = fmaxf(0.f, fmaxf(bl - v, v - bh)), gc = fmaxf(0.f, fmaxf(cl - v, v - ch));
                const float g = fmaxf(0.f, fmaxf(cl - bh, bl - ch));
                pb = fmaf(gb, gb, pb);
                pc = fmaf(gc, gc, pc);
                bc = fmaf(g, g, bc);
            }
        };
        const bool resident = __popc(S.mask) <= TRI_GROUP_A;
        if (threadIdx.x < nr * TILE) {
            const float4 pi = PA[threadIdx.x];
            float ij2, ik2, jk2;
            bounds2(pi, [&](int a) { return S.box[0][a]; }, [&](int a) { return S.box[0][3 + a]; }, S.box[1], ij2, ik2, jk2);
            const bool keep = (int)(threadIdx.x % TILE) < S.meta[threadIdx.x / TILE].y &&
                              (p.tame ? possible(ij2, ik2, jk2) : !(fmaxf(ij2, ik2) > reach2));
            const unsigned b = __ballot_sync(0xffffffffu, keep);
            int at = 0;
            if (lane == 0 && b) at = atomicAdd(&S.end_i, __popc(b));
            at = __shfl_sync(0xffffffffu, at, 0);
            if (keep) S.list[at + __popc(b & ((1u << lane) - 1u))] = (uint8_t)threadIdx.x;
            if (b && resident) box_add(S.abox, lane, keep, pi, pi);
        }
        if (ch == 0 && !resident && warp == TRI_WARPS - 1) {
            const bool has = (S.mask >> lane) & 1u;
            const size_t a = 2 * (size_t)(unit.y + (has ? lane : __ffs(S.mask) - 1));
            box_add(S.abox, lane, has, J.box[0][a], J.box[0][a + 1]);
        }
        __syncthreads();
        if (S.end_i == 0) continue;
        if (!have_jk) {
            have_jk = true;
            // The points j and k likewise, with the box of the listed i in place
            // of the other's tile, and moved to the front of their tiles in
            // order; their places there are j and k from here on.  (Where B and
            // C are one tile both tests are the same, so k > j stays as it is.)
            // A unit of 100 voxels has 14 points i on average: its 64 x 64 j-k
            // sides cost more than its i.  (Kernel 2.56 -> 2.35 ms, 10k-point
            // estimator 10.0 -> 9.9.)
            if (warp < 2) {
                float4* pts = warp == 0 ? PB : PC;
                const float* other = S.box[1 - warp];
                const int n = warp == 0 ? numB : numC;
                const float4 p0 = pts[lane], p1 = pts[lane + 32];
                auto keep = [&](float4 pt) {
                    float pi2, jk2, io2;
                    bounds2(pt, [&](int a) { return ordered_float(S.abox[a]); },
                            [&](int a) { return ordered_float(S.abox[3 + a]); }, other, pi2, jk2, io2);
                    return !p.tame || possible(pi2, jk2, io2);
                };
                const bool k0 = lane < n && keep(p0), k1 = lane + 32 < n && keep(p1);
                const unsigned b0 = __ballot_sync(0xffffffffu, k0), b1 = __ballot_sync(0xffffffffu, k1);
                const unsigned lt = (1u << lane) - 1u;
                uint8_t* list = warp == 0 ? S.jlist : S.klist;
                if (k0) {
                    pts[__popc(b0 & lt)] = p0;
                    list[__popc(b0 & lt)] = (uint8_t)lane;
                }
                if (k1) {
                    pts[__popc(b0) + __popc(b1 & lt)] = p1;
                    list[__popc(b0) + __popc(b1 & lt)] = (uint8_t)(lane + 32);
                }
                if (lane == 0) (warp == 0 ? S.nj : S.nk) = __popc(b0) + __popc(b1);
            }
            __syncthreads();
            numB = S.nj;
            numC = S.nk;
            key_k0 = pkey(PC[lane]);
            key_k1 = pkey(PC[lane + 32]);
            // rows j of the j-k side table and their class sets, one warp per row
            for (int j = warp; j < numB; j += TRI_WARPS) {
                const float4 pj = PB[j];
                int c0 = 0, c1 = 0;
                if (lane < numC) {
                    float d = ref_dist<false>(pj, PC[lane]);
                    int w = tri_side_word<MODE>(d, p);
                    JKd[j * TILE + lane] = d;
                    JKw[j * TILE + lane] = (short)w;
                    c0 = side_class<MODE>(w, d, p);
                }
                if (lane + 32 < numC) {
                    float d = ref_dist<false>(pj, PC[lane + 32]);
                    int w = tri_side_word<MODE>(d, p);
                    JKd[j * TILE + lane + 32] = d;
                    JKw[j * TILE + lane + 32] = (short)w;
                    c1 = side_class<MODE>(w, d, p);
                }
                side_sets(JM + j, TILE, lane, c0, c1);
                const int kj = pkey(pj);
                const unsigned long long kge = ballot64(lane < numC && key_k0 >= kj, lane + 32 < numC && key_k1 >= kj);
                if (lane == 0) JM[JM_KEY * TILE + j] = kge;
            }
            __syncthreads();
        }
        for (;;) {
            // points of the chunk's A tiles are handed out to warps
            // dynamically (balances the very uneven work per point)
            int ii = 0;
            if (lane == 0) ii = atomicAdd(&S.next_i, 1);
            ii = __shfl_sync(0xffffffffu, ii, 0);
            if (ii >= S.end_i) break;
            ii = S.list[ii];
            const int4 meta = S.meta[ii / TILE];
            const int i = ii % TILE;
            // in a diagonal tile pair j > i; else every j
            const int j_after = meta.z ? i + meta.w : -1;
            const float4 pi = PA[ii];
            const int ki = pkey(pi);
            // i-k sides: words for the binning path, class masks for the filter
            int c0 = 0, c1 = 0;
            if (lane < numC) {
                float d = ref_dist<false>(pi, PC[lane]);
                int w = tri_side_word<MODE>(d, p);
                row_ik[lane] = make_int2(__float_as_int(d), w);
                c0 = side_class<MODE>(w, d, p);
            }
            if (lane + 32 < numC) {
                float d = ref_dist<false>(pi, PC[lane + 32]);
                int w = tri_side_word<MODE>(d, p);
                row_ik[lane + 32] = make_int2(__float_as_int(d), w);
                c1 = side_class<MODE>(w, d, p);
            }
            const unsigned long long any_k = side_sets(sets, 1, lane, c0, c1);
            if (!any_k) continue;  // no k within reach of i (warp-uniform)
            __syncwarp();
            const uint32_t pred = S.pred;
            unsigned long long kge_i = 0;  // PRED_DDR: key_k >= key_i; PRED_RDD: key_k <= key_i
            if (!UNIT && pred == PRED_DDR) kge_i = ballot64(lane < numC && key_k0 >= ki, lane + 32 < numC && key_k1 >= ki);
            if (!UNIT && pred == PRED_RDD) kge_i = ballot64(lane < numC && key_k0 <= ki, lane + 32 < numC && key_k1 <= ki);
            // i-j sides: words for the binning path; each lane then forms the
            // candidate-k mask of its own two j's (the scan over j is lane-parallel)
            // mask of candidate k's (and of weight-2 k's) of the pair (i, j)
            auto scan_j = [&](int j, unsigned long long& cm, unsigned long long& w2) -> bool {
                cm = 0;
                w2 = 0;
                if (j >= numB) return false;
                float d = ref_dist<false>(pi, PB[j]);
                int w = tri_side_word<MODE>(d, p);
                row_ij[j] = make_int2(__float_as_int(d), w);
                const int c = side_class<MODE>(w, d, p);
                bool ok = c != 0 && any_k && (int)S.jlist[j] > j_after;
                if (UNIT && pred == PRED_SAME) ok = ok && ki <= pkey(PB[j]);
                if (!ok) return false;
                cm = candidate_mask(c, sets, JM + j);
                if (diag_jk) cm &= j >= 63 ? 0ull : (~0ull << (j + 1));
                if (!UNIT && pred == PRED_RDD) {
                    // weight [key_j <= key_i] + [key_k <= key_i]
                    if (pkey(PB[j]) <= ki) {
                        w2 = cm & kge_i;
                    } else {
                        cm &= kge_i;
                    }
                } else if (!UNIT || pred != PRED_NONE) {
                    const unsigned long long kge_j = JM[JM_KEY * TILE + j];
                    if (!UNIT) {
                        w2 = cm & kge_i & kge_j;  // weight 2: k >= i and k >= j
                        cm &= kge_i | kge_j;      // weight 0 otherwise
                    } else {
                        cm &= kge_j;              // key_j <= key_k
                    }
                }
                return true;
            };
            // (one copy of the scan: 100 voxels 1.99 -> 1.91 ms)
            unsigned long long cm0 = 0, w20 = 0, cm1 = 0, w21 = 0;
            int nok = 0;
#pragma unroll 1
            for (int h = 0; h < numB; h += 32) {
                cm0 = cm1, w20 = w21;
                nok += __popc(__ballot_sync(0xffffffffu, scan_j(lane + h, cm1, w21)));
            }
            if (numB <= 32) cm0 = cm1, cm1 = 0, w20 = w21;
            // walked (i, j, k): every k with a usable i-k side, for every usable j
            ev += (unsigned)__popcll(any_k) * (unsigned)nok;
            __syncwarp();
            const uint32_t ia = (uint32_t)(meta.x + i);
            // Candidates of this i: every j with a non-empty mask in turn, expanded
            // by the whole warp (lanes over k), queued and binned 64 at a time.
            // (A lane-parallel compaction of the j's with few candidates, through
            // a prefix sum of per-lane counts, measured slower on clustered data:
            // its scattered j/k break the conflict-free table reads of binning.)
            const unsigned lbit = 1u << lane, lt = lbit - 1u;
            // queue entries of this lane's k = lane and k = lane + 32 (weight 1;
            // plus j and the weight bit of two-array jobs)
            const uint32_t klo = ((uint32_t)lane << 6) | (1u << 12), khi = ((uint32_t)(lane + 32) << 6) | (1u << 12);
            int qn = 0;  // queued candidates (warp-uniform)
            unsigned live = __ballot_sync(0xffffffffu, cm0 != 0ull), live1 = __ballot_sync(0xffffffffu, cm1 != 0ull);
            uint32_t j0 = 0;  // (one place that bins, for the code's size)
            for (;;) {
                if (live) {
                    const int src = __ffs(live) - 1;
                    live &= live - 1u;
                    const uint32_t j = (uint32_t)src + j0;
                    const unsigned lo = __shfl_sync(0xffffffffu, (unsigned)cm0, src);
                    const unsigned hi = __shfl_sync(0xffffffffu, (unsigned)(cm0 >> 32), src);
                    uint32_t vlo = klo + j, vhi = khi + j;
                    if (!UNIT) {
                        const unsigned w2lo = __shfl_sync(0xffffffffu, (unsigned)w20, src);
                        const unsigned w2hi = __shfl_sync(0xffffffffu, (unsigned)(w20 >> 32), src);
                        vlo += (w2lo & lbit) ? (1u << 12) : 0u;
                        vhi += (w2hi & lbit) ? (1u << 12) : 0u;
                    }
                    const int nlo = __popc(lo);
                    if (lo & lbit) cand[qn + __popc(lo & lt)] = (Entry)vlo;
                    if (hi & lbit) cand[qn + nlo + __popc(hi & lt)] = (Entry)vhi;
                    qn += nlo + __popc(hi);
                    if (qn < 64) continue;
                } else if (live1) {
                    live = live1, live1 = 0;
                    j0 = 32;
                    cm0 = cm1, w20 = w21;
                    continue;
                } else if (qn == 0) {
                    break;
                }
                const int n = min(qn, 64);
                __syncwarp();
                qn -= n;
                run_candidates<THETA_FULL, MODE, UNIT>(cand + qn, n, row_ij, row_ik, JKd, JKw, p, Hw, q, S, ia);
                bn += n;
                __syncwarp();
            }
            __syncwarp();
        }
    }
    // (per-warp totals into the CTA's counters: no 64-bit accumulators live
    // in registers across the kernel)
    if (lane == 0) {
        atomicAdd(&evaluated, (unsigned long long)ev);
        atomicAdd(&binned, (unsigned long long)bn);
    }
}

#ifndef TRI_MIN_BLOCKS
#define TRI_MIN_BLOCKS 4
#endif
// Persistent over the plan's units: tiles B and C of a job with a mask of A
// tiles.
template <bool THETA_FULL, int MODE, typename Entry>
__global__ void __launch_bounds__(TRI_THREADS, TRI_MIN_BLOCKS)
triangle_fast_kernel(const DevJob* __restrict__ jobs, UnitList ul, unsigned int* counter, TriParams p, RecheckQueue q,
                     int copies) {
    extern __shared__ __align__(16) unsigned char smem[];
    float4* P = reinterpret_cast<float4*>(smem);
    unsigned long long* JM = reinterpret_cast<unsigned long long*>(P + (2 + TRI_GROUP_A) * TILE);
    int2* IJ = reinterpret_cast<int2*>(JM + JM_WORDS * TILE + TRI_WARPS * SET_WORDS);
    int2* IK = IJ + TRI_WARPS * TILE;
    float* JKd = reinterpret_cast<float*>(IK + TRI_WARPS * TILE);
    Entry* Q = reinterpret_cast<Entry*>(JKd + TILE * TILE);
    short* JKw = reinterpret_cast<short*>(Q + TRI_WARPS * TRI_QCAP);
    unsigned int* H = reinterpret_cast<unsigned int*>(JKw + TILE * TILE);
    __shared__ TriShared S;
    for (int b = threadIdx.x; b < copies * p.len; b += blockDim.x) H[b] = 0;
    unsigned int* Hw = H + ((threadIdx.x >> 5) % copies) * p.len;
    int cur = -1;
    unsigned int since = 0;
    __shared__ unsigned long long ev, bn;  // triangles walked and binned by this CTA
    if (threadIdx.x == 0) ev = bn = 0;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) {
            const unsigned int t = atomicAdd(counter, 1u);
            const bool any = t < ul.n && ul.u0 + t < ul.header->nunits;
            S.unit = any ? ul.units[ul.u0 + t] : make_uint4(TASK_NONE, 0, 0, 0);
            S.mask = any ? ul.masks[ul.u0 + t] : 0u;
            if (any) S.pred = jobs[S.unit.x & UNIT_SLOT_MASK].mode & JOB_PRED_MASK;
        }
        __syncthreads();
        if (S.unit.x == TASK_NONE) break;
        const int slot = (int)(S.unit.x & UNIT_SLOT_MASK);
        // (a unit holds at most MAX_WINDOW <= FLUSH_EVERY tile triples)
        const unsigned int n = __popc(S.mask);
        if ((slot != cur || since + n > FLUSH_EVERY) && cur >= 0) {
            flush_hist(H, copies, p.len, jobs[cur].hist);
            since = 0;
        }
        cur = slot;
        since += n;
        if (n == 0) continue;  // a part without A tiles
        if (S.pred == PRED_DDR || S.pred == PRED_RDD)
            triangle_group_fast<false, THETA_FULL, MODE, Entry>(jobs, p, P, JKd, JKw, IJ, IK, Q, JM, S, Hw, q, ev, bn);
        else
            triangle_group_fast<true, THETA_FULL, MODE, Entry>(jobs, p, P, JKd, JKw, IJ, IK, Q, JM, S, Hw, q, ev, bn);
    }
    if (cur >= 0) flush_hist(H, copies, p.len, jobs[cur].hist);
    __syncthreads();
    if (threadIdx.x == 0) {
        if (ev) atomicAdd(q.evaluated, ev);
        if (bn) atomicAdd(q.evaluated + 1, bn);
    }
}

// ---------------------------------------------------------------------------
// Triangle parametrizations from neighbour lists.
//
// Each triangle is taken at one of its points, the centre: the one opposite its
// longest side, so that the centre's two sides are the shortest S and the
// middle M (equal longest sides: the first of the points concerned in (rank,
// position) order, sides compared as the reference's floats).  A counted
// triangle has S < s_hi and M below a limit of S (q_hi S, 1/q_lo S for JBJ, or
// s_hi): for a centre the points within s_hi ("near") make J lists, all points
// within the largest limit K lists, and a pair (j, k) whose third side is the
// longest is a triangle.  One warp per centre, lists of 64 in shared memory
// filled in the order of the views' tiles and used up in turn, pairs tested
// eight to a lane, and what passes queued and binned two to a lane.  No
// barrier but where the CTA's shared histogram changes hands.
//
// Issue-bound: 14 lane-instructions a tested pair, 29 to queue what passes (of
// 32), some 250 to fetch, test and bin one.  Against tile triples
// (triangle_group_fast) it wins where those have few CTAs, or few near
// triangles (run_group has the rule and the times).  Tried and left: two
// triangles a lane in packed instructions (500 instructions a batch of 64, no
// faster), marks kept by each lane and binned one a round instead of a queue
// (30 % of the lanes idle: 10k-point blobs 14.3 -> 16.7 ms), 32 warps of 64
// registers instead of 24 of 80 (17.4 against 15.3 ms), a CTA barrier per change
// of output slot (all slots' histograms are resident where they fit).

constexpr int TL_LIST = 64;  // entries of a list
constexpr int TL_QCAP = 288;  // queued pairs: up to 31 pending + 256 of one step
constexpr unsigned TL_SPILL = 1u << 28;
constexpr int TL_TILES = 64;  // near tiles kept per list (more: found again at every pass)
// Margin of compared squares beside their relative ones: subnormal squares (the
// smallest number is 1.4e-45) have lost bits, in other places in the reference's
// sums than in the fused ones here.
constexpr float TL_TINY2 = 2e-38f;

struct TriListWarp {
    // lists J (0) and K (1)
    float x[2][TL_LIST], y[2][TL_LIST], z[2][TL_LIST], d[2][TL_LIST];
    int code[2][TL_LIST];
    uint32_t pos[2][TL_LIST];
    float lim[TL_LIST];  // J: squared limit of the middle side
    uint16_t queue[TL_QCAP];
    uint32_t tiles[2][TL_TILES];
    unsigned int dump[32];
    uint4 item;          // job, first centre, centres, part
};

size_t tri_list_smem_bytes(int hist_len, int hists, int warps) {
    return (size_t)warps * sizeof(TriListWarp) + (size_t)hist_len * hists * 4;
}

// Which points of a view a list takes.
constexpr int TL_NEAR = 1, TL_FAR = 2;

// A bin coordinate (minus 0.5) as the bits of coordinate + MAGIC (bin =
// bits - MAGIC_BITS) and its distance from the bin's centre.
__device__ __forceinline__ uint32_t magic_bits(float f, float& e) {
    const float tm = __fadd_rn(f, MAGIC);
    e = __fsub_rn(f, __fsub_rn(tm, MAGIC));
    return __float_as_uint(tm);
}

// The angle's coordinate of theta_fast2 for one cosine; t: 1 - |c|, y: its
// reciprocal square root.
__device__ __forceinline__ void theta_fast(float c, const TriParams& p, float& f, float& t, float& y) {
    const float x = fabsf(c);
    t = __fsub_rn(1.0f, x);
    y = rsqrt_approx(t);
    const float sq = __fmul_rn(t, y);
    float P = fmaf(p.t_coef[5], x, p.t_coef[4]);
    P = fmaf(P, x, p.t_coef[3]);
    P = fmaf(P, x, p.t_coef[2]);
    P = fmaf(P, x, p.t_coef[1]);
    P = fmaf(P, x, p.t_coef[0]);
    const float a = fmaf(sq, P, -p.t_half);
    f = __int_as_float(__float_as_int(a) ^ (__float_as_int(c) & 0x80000000)) + p.t_off0;
}

// Bins a triangle of weight w (0: none) with sides s <= m <= l (l2: about the
// square of l) and the s-bin codes of s and m; true where it has to be
// recomputed exactly.  One triangle a lane: two in packed instructions took 500
// instructions a batch of 64 here, spilled registers among them.
//
// s and m are the reference's floats, l2 a fused sum of the same differences.
// With u = 2^-24 the numerator of a cosine is within 13 u of the sum of the
// squares of the reference's and its reciprocal denominator within 8 u, so the
// cosine within 21 u E = 1.25e-6 E, E = (s^2 + m^2 + l^2) / (2 s m): the guard
// takes 1.5e-6 E, moves an angle by at most 1.42 times that over sqrt(1 - |c|),
// and a cosine within twice that of +-1 is always recomputed.  Ratios of l are
// within 15 u.  (The double-precision geometry: see triangle_full2.)
template <int MODE>
__device__ __forceinline__ bool tri_list_bin(float s, float m, float l2, int cs, int cm, unsigned w, const TriParams& p,
                                             uint32_t base, uint32_t none) {
    const bool v02 = w && (unsigned)cs < (unsigned)p.S;  // shortest side in range
    const bool v1 = w && (unsigned)cm < (unsigned)p.S;   // middle side in range
    const float rs = rcp_approx(s), rm = rcp_approx(m), rl = rsqrt_approx(l2), l = l2 * rl;
    // address of (code, q bits, t bits): both MAGIC_BITS folded into the base
    const uint32_t Q = (uint32_t)p.Q, T4 = 4u * (uint32_t)p.T;
    const uint32_t at = base - (uint32_t)MAGIC_BITS * (T4 + 4u);
    if (MODE == FAST_JBJ) {
        float e1, e2;
        const uint32_t b1 = magic_bits(fmaf(s * rm, p.q_scale, p.q_off), e1);
        const uint32_t b2 = magic_bits(fmaf((l - m) * rs, p.t_coef[0], p.t_off0), e2);
        // (l - m cancels: its error is 8 u l / s)
        const bool safe = fabsf(e1) <= p.q_thr && fabsf(e2) <= fmaf(-p.list_t, l * rs, p.t_thrA);
        const bool take = v02 && safe && b1 - MAGIC_BITS < Q && b2 - MAGIC_BITS < (uint32_t)p.T;
        count_at<false>(take ? ((uint32_t)cs * Q + b1) * T4 + (4u * b2 + at) : none, w);
        return v02 && !safe;
    }
    const float s2 = s * s, m2 = m * m;
    const float rsq = rs * p.q_scale, rmq = rm * p.q_scale, hsm = rs * rm * 0.5f, hml = rm * rl * 0.5f;
    const float sm2 = s2 + m2;
    float q0e, q1e, q2e, t0e, t1e, t2e;
    const uint32_t q0 = magic_bits(fmaf(m, rsq, p.q_off), q0e), q1 = magic_bits(fmaf(l, rmq, p.q_off), q1e),
                   q2 = magic_bits(fmaf(l, rsq, p.q_off), q2e);
    float f0, f1, thr0, thr1, tc0, tc1, y0, y1;
    theta_fast((sm2 - l2) * hsm, p, f0, tc0, y0);
    theta_fast((m2 - s2 + l2) * hml, p, f1, tc1, y1);
    const float sum2 = sm2 + l2, E0 = sum2 * hsm, E1 = sum2 * hml;
    constexpr float close = MODE == FAST_GEOM ? 8e-6f : 3e-6f;
    thr0 = tc0 > close * E0 ? fmaf(-p.list_t, E0 * y0, p.t_thrA) : -1.f;
    thr1 = tc1 > close * E1 ? fmaf(-p.list_t, E1 * y1, p.t_thrA) : -1.f;
    bool us = true, um = true;
    if (MODE == FAST_GEOM) {
        float es, em;
        magic_bits(fmaf(s, p.geo_s_inv, p.geo_s_off), es);
        magic_bits(fmaf(m, p.geo_s_inv, p.geo_s_off), em);
        us = fabsf(es) <= p.geo_s_thr;
        um = fabsf(em) <= p.geo_s_thr;
    }
    const uint32_t t0 = magic_bits(f0, t0e), t1 = magic_bits(f1, t1e),
                   t2 = magic_bits(p.t2_off - f0 - f1, t2e);
    const bool u02 = fabsf(q0e) <= p.list_q_thr && fabsf(t0e) <= thr0 && fabsf(q2e) <= p.list_q_thr &&
                     fabsf(t2e) <= thr0 + thr1 + (-0.5f - 1e-6f) && us;
    const bool u1 = fabsf(q1e) <= p.list_q_thr && fabsf(t1e) <= thr1 && um;
    const bool guard = (v02 && !u02) || (v1 && !u1);
    const bool n02 = v02 && !guard, n1 = v1 && !guard;
    const uint32_t T = (uint32_t)p.T, rs0 = (uint32_t)cs * Q, rm0 = (uint32_t)cm * Q;
    const bool ok0 = n02 && q0 - MAGIC_BITS < Q && t0 - MAGIC_BITS < T;
    const bool ok1 = n1 && q1 - MAGIC_BITS < Q && t1 - MAGIC_BITS < T;
    const bool ok2 = n02 && q2 - MAGIC_BITS < Q && t2 - MAGIC_BITS < T;
    count_at<false>(ok0 ? (rs0 + q0) * T4 + (4u * t0 + at) : none, w);
    count_at<false>(ok1 ? (rm0 + q1) * T4 + (4u * t1 + at) : none, w);
    count_at<false>(ok2 ? (rs0 + q2) * T4 + (4u * t2 + at) : none, w);
    return guard;
}

// One warp's centre: its job, its point, and the running state of its lists.
template <int MODE>
struct TriCentre {
    const DevJob& J;
    const TriParams& p;
    TriListWarp& W;
    const RecheckQueue& rq;
    const uint32_t base;
    const uint32_t slot;
    float4 c;
    uint32_t cpos;
    int near0, near1;  // near tiles of each list's view
    __device__ __forceinline__ int ntl(int v) const { return v ? near1 : near0; }
    int qn = 0;       // queued pairs
    unsigned tested = 0, binned = 0, accounted = 0;
    unsigned int *H, *since;  // the CTA's histograms and triangles since they were flushed
    unsigned long long* out;  // where they are flushed to
    int nbins;
    int lane;

    __device__ __forceinline__ TriCentre(const DevJob& J_, const TriParams& p_, TriListWarp& W_, const RecheckQueue& rq_,
                                         unsigned int* H_, int hists, unsigned int* since_, uint32_t slot_)
        : J(J_), p(p_), W(W_), rq(rq_),
          base(shared_addr(H_) + (hists == 1 ? 0u : 4u * (uint32_t)(J_.weight >> 32) * (uint32_t)p_.len)), slot(slot_),
          H(H_), since(since_), out(hists == 1 ? J_.hist : rq_.hists), nbins(hists * p_.len), lane(threadIdx.x & 31) {}

    __device__ __forceinline__ bool near_box(const float4* bx) const {
        const float4 lo = bx[0], hi = bx[1];
        const float gx = fmaxf(0.f, fmaxf(lo.x - c.x, c.x - hi.x)), gy = fmaxf(0.f, fmaxf(lo.y - c.y, c.y - hi.y)),
                    gz = fmaxf(0.f, fmaxf(lo.z - c.z, c.z - hi.z));
        return (gx * gx + gy * gy + gz * gz) * (1.0f - 4e-5f) < p.list_r2;
    }
    // near tiles of view v (role 1 + v)
    __device__ __forceinline__ int find_tiles(int v) {
        int n = 0;
        for (int t0 = 0; t0 < J.ntiles[1 + v]; t0 += 32) {
            const bool near = t0 + lane < J.ntiles[1 + v] && near_box(J.box[1 + v] + 2 * (size_t)(t0 + lane));
            const unsigned m = __ballot_sync(0xffffffffu, near);
            const int at = n + __popc(m & ((1u << lane) - 1u));
            if (near && at < TL_TILES) W.tiles[v][at] = (uint32_t)(t0 + lane);
            n += __popc(m);
        }
        __syncwarp();
        return n;
    }
    // Steps (half tiles) of view v before `end` (even): the tile of step s,
    // advancing s past tiles out of reach where the near tiles are not kept; -1
    // (s = end) where none is left.  s never goes back: an even s moves to the
    // first half of a tile at or after it, an odd s stays.
    __device__ __forceinline__ int tile_at(int v, int end, int& s) const {
        if (s >= end) return -1;
        if (ntl(v) <= TL_TILES) return (int)W.tiles[v][s >> 1];
        if (s & 1) return s >> 1;  // (its first half found it)
        for (int t0 = s >> 1; 2 * t0 < end; t0 += 32) {
            const bool near = 2 * (t0 + lane) < end && near_box(J.box[1 + v] + 2 * (size_t)(t0 + lane));
            const unsigned m = __ballot_sync(0xffffffffu, near);
            if (m) {
                const int t = t0 + __ffs(m) - 1;
                s = 2 * t;
                return t;
            }
        }
        s = end;
        return -1;
    }
    // Fills list h (0: J, 1: K) from view v's steps s on, with the points of
    // `which` (near points only from step `near_from` on), until it may not
    // hold the next step or step `end` is reached; returns the entries.
    __device__ __forceinline__ int fill(int h, int v, int which, int near_from, int end, int& s) {
        int n = 0;
        for (;;) {
            const int t = tile_at(v, end, s);
            if (t < 0 || n + 32 > TL_LIST) break;
            const int b0 = J.tile_start[1 + v][t] + 32 * (s & 1), b1 = J.tile_start[1 + v][t + 1];
            const bool with_near = (which & TL_NEAR) && s >= near_from;
            s++;
            const uint32_t pos = (uint32_t)(b0 + lane);
            float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
            float d = 0.f;
            bool in = b0 + lane < b1;
            if (in) {
                q = J.pts[1 + v][pos];
                const float dx = __fsub_rn(c.x, q.x), dy = __fsub_rn(c.y, q.y), dz = __fsub_rn(c.z, q.z);
                const float d2 = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
                in = d2 < p.list_r2;
                if (in) d = __fsqrt_rn(d2);
            }
            const float s_top = MODE == FAST_GEOM ? p.geo_s_above : p.s_hi;
            // zero sides count nowhere (the geometry's double length may not be zero: the
            // centre itself apart, they stay); JBJ: nor do sides below s_lo
            if (MODE == FAST_JBJ) in = in && d >= p.s_lo && d > 0.f;
            else if (MODE == FAST_GEOM) in = in && !(pos == cpos && J.pts[1 + v] == J.pts[0]);
            else in = in && d > 0.f;
            in = in && (d < s_top ? with_near : (which & TL_FAR) != 0);
            const unsigned m = __ballot_sync(0xffffffffu, in);
            if (in) {
                const int at = n + __popc(m & ((1u << lane) - 1u));
                int code = CODE16_ABOVE;
                if (MODE == FAST_GEOM) {
                    if (d < p.geo_s_below) code = CODE16_BELOW;
                    else if (d < s_top) code = min(max(__float2int_rz(__fdiv_rn(__fsub_rn(d, p.s_lo), p.s_bw)), 0), p.S - 1);
                } else if (d < p.s_lo) {
                    code = CODE16_BELOW;
                } else if (d < s_top) {
                    code = __float2int_rz(__fdiv_rn(__fsub_rn(d, p.s_lo), p.s_bw));
                }
                W.x[h][at] = q.x;
                W.y[h][at] = q.y;
                W.z[h][at] = q.z;
                W.d[h][at] = d;
                W.code[h][at] = code;
                W.pos[h][at] = pos;
                if (h == 0) {
                    const float lim = fmaxf(d * p.list_q, p.list_top);
                    W.lim[at] = fmaf(lim, lim, TL_TINY2);
                }
            }
            n += __popc(m);
        }
        // padding to whole groups of four
        if (h == 0 && lane < 4 && n + lane < ((n + 3) & ~3)) {
            W.x[0][n + lane] = W.y[0][n + lane] = W.z[0][n + lane] = 0.f;
            W.d[0][n + lane] = 0.f;
            W.lim[n + lane] = -1.f;
        }
        __syncwarp();
        return n;
    }
    // (rank, position) order of two points
    static __device__ __forceinline__ bool first_of(uint32_t ra, uint32_t pa, uint32_t rb, uint32_t pb) {
        return ra < rb || (ra == rb && pa < pb);
    }
    // Bins queue entries [at, at + n), n <= 32.  kh: the list that k comes from
    // (0 in pairs of one list); vj, vk: the views of j and k.
    __device__ __forceinline__ void run(int at, int n, int kh, int vj, int vk) {
        __syncwarp();
        const bool any = lane < n;
        const uint32_t e = any ? (uint32_t)W.queue[at + lane] : 0u;
        const int j = e & 63, k = e >> 6;
        const float4 a = make_float4(W.x[0][j], W.y[0][j], W.z[0][j], 0.f);
        const float4 b = make_float4(W.x[kh][k], W.y[kh][k], W.z[kh][k], 0.f);
        const float dj = W.d[0][j], dk = W.d[kh][k];
        const int cj = W.code[0][j], ck = W.code[kh][k];
        const float s = fminf(dj, dk), m = fmaxf(dj, dk);
        const float dx = a.x - b.x, dy = a.y - b.y, dz = a.z - b.z, l2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
        const float m2 = m * m;
        bool take = any && l2 > m2;
        if (any && fabsf(l2 - m2) <= fmaf(2e-6f, m2, TL_TINY2)) {
            // too close to tell: the reference's floats
            const float l = ref_dist<false>(a, b);
            take = l >= m && (MODE == FAST_GEOM || l > 0.f);
            if (take && l == m) {
            // equal longest sides: j lies opposite k's side, k opposite j's
            const uint32_t rc = J.mode >> TL_RANK_SHIFT & 3u, r1 = J.mode >> (TL_RANK_SHIFT + 2 + 2 * vj) & 3u,
                           r2 = J.mode >> (TL_RANK_SHIFT + 2 + 2 * vk) & 3u;
            if (dk == m) take = first_of(rc, cpos, r1, W.pos[0][j]);
            if (dj == m) take = take && first_of(rc, cpos, r2, W.pos[kh][k]);
            }
        }
        unsigned w = take ? 1u : 0u;
        const uint32_t pred = J.mode & JOB_PRED_MASK;
        if (pred != PRED_NONE && take) {
            // keys in the reference's roles
            int key[3] = {0, 0, 0};
            const int kc = pkey(c), kj = pkey(J.pts[1 + vj][W.pos[0][j]]), kk = pkey(J.pts[1 + vk][W.pos[kh][k]]);
            const uint32_t oc = J.mode >> TL_ROLE_SHIFT & 3u, o1 = J.mode >> (TL_ROLE_SHIFT + 2 + 2 * vj) & 3u,
                           o2 = J.mode >> (TL_ROLE_SHIFT + 2 + 2 * vk) & 3u;
#pragma unroll
            for (int r = 0; r < 3; r++) key[r] = (uint32_t)r == oc ? kc : (uint32_t)r == o1 ? kj : (uint32_t)r == o2 ? kk : 0;
            if (pred == PRED_DDR) w = (unsigned)(key[2] >= key[0]) + (unsigned)(key[2] >= key[1]);
            else if (pred == PRED_SAME) w = key[0] <= key[1] && key[1] <= key[2] ? 1u : 0u;
            else w = key[1] <= key[2] ? 1u : 0u;
        }
        // (a longest side whose square may have lost bits to underflow: 0 is in every band)
        const bool guard = tri_list_bin<MODE>(s, m, l2 < 1e-36f ? 0.f : l2, min(cj, ck), max(cj, ck), w, p, base,
                                              shared_addr(W.dump + lane));
        if (guard) {  // (positions in the job's order of views)
            const uint32_t pj = W.pos[0][j], pk = W.pos[kh][k];
            push_recheck(rq, slot, w, cpos, vj < vk ? pj : pk, vj < vk ? pk : pj);
        }
        binned += (unsigned)n;
        __syncwarp();
    }
    // Tests the pairs of J's nj entries with nk entries of list kh (0: of J
    // itself, j < k) and bins those whose third side is the longest.  vj, vk:
    // the views of j and k (0 and 1 also where both are one).
    __device__ __forceinline__ void pairs(int nj, int nk, int kh, int vj, int vk) {
        const unsigned lt = (1u << lane) - 1u;
        f32x2 X[2], Y[2], Z[2];
        float d2[2], dm[2];
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const int k = lane + 32 * r;
            const bool in = k < nk;
            X[r] = splat2(in ? W.x[kh][k] : 0.f);
            Y[r] = splat2(in ? W.y[kh][k] : 0.f);
            Z[r] = splat2(in ? W.z[kh][k] : 0.f);
            const float d = in ? W.d[kh][k] : 3e18f;  // (past every limit)
            d2[r] = d * d;
            dm[r] = fmaf(d2[r], 1.0f - 1e-5f, -TL_TINY2);
        }
        const bool two = nk > 32;
        const uint32_t kj = (uint32_t)lane << 6, qbase = shared_addr(W.queue);
        tested += (unsigned)(kh == 0 ? nj * (nj - 1) / 2 : nj * nk);
        for (int j = 0; j < nj; j += 4) {
            const float4 x4 = *reinterpret_cast<const float4*>(W.x[0] + j), y4 = *reinterpret_cast<const float4*>(W.y[0] + j),
                         z4 = *reinterpret_cast<const float4*>(W.z[0] + j), d4 = *reinterpret_cast<const float4*>(W.d[0] + j),
                         l4 = *reinterpret_cast<const float4*>(W.lim + j);
            const f32x2 xj[2] = {pk2(x4.x, x4.y), pk2(x4.z, x4.w)}, yj[2] = {pk2(y4.x, y4.y), pk2(y4.z, y4.w)},
                        zj[2] = {pk2(z4.x, z4.y), pk2(z4.z, z4.w)}, dj[2] = {pk2(d4.x, d4.y), pk2(d4.z, d4.w)};
            const float lj[4] = {l4.x, l4.y, l4.z, l4.w};
            float mj[4];
            const f32x2 part = splat2(1.0f - 1e-5f), tiny = splat2(-TL_TINY2);
            up2(fma2(mul2(dj[0], dj[0]), part, tiny), mj[0], mj[1]);
            up2(fma2(mul2(dj[1], dj[1]), part, tiny), mj[2], mj[3]);
#pragma unroll
            for (int r = 0; r < 2; r++) {
                if (r == 1 && !two) continue;  // warp-uniform
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const f32x2 dx = sub2(xj[h], X[r]), dy = sub2(yj[h], Y[r]), dz = sub2(zj[h], Z[r]);
                    float L2[2];
                    up2(fma2(dz, dz, fma2(dy, dy, mul2(dx, dx))), L2[0], L2[1]);
#pragma unroll
                    for (int t = 0; t < 2; t++) {
                        const int q = 2 * h + t;
                        const bool ok = L2[t] >= fmaxf(mj[q], dm[r]) && d2[r] < lj[q] && (kh != 0 || j + q < lane + 32 * r);
                        const unsigned m = __ballot_sync(0xffffffffu, ok);
                        store_if(ok, qbase + 2u * (uint32_t)(qn + __popc(m & lt)), kj + (uint32_t)(j + q + (r << 11)));
                        qn += __popc(m);
                    }
                }
            }
            // full batches; after the last step also the rest
            const int least = j + 4 < nj ? 32 : 1;
            while (qn >= least) {
                const int n = min(qn, 32);
                qn -= n;
                run(qn, n, kh, vj, vk);
            }
        }
        // a triangle adds at most six to one bin (three permutations, weight
        // two): the warp that brings the CTA to 2^28 triangles empties the
        // 32-bit counters while the others count on
        const unsigned b1 = binned - accounted;
        if (b1) {
            unsigned before = 0;
            if (lane == 0) before = atomicAdd(since, b1);
            before = __shfl_sync(0xffffffffu, before, 0);
            if (before < TL_SPILL && before + b1 >= TL_SPILL) {
                for (int b = lane; b < nbins; b += 32) {
                    const unsigned int v = atomicExch(H + b, 0u);
                    if (v) atomicAdd(out + b, (unsigned long long)v);
                }
                if (lane == 0) atomicSub(since, before + b1);
            }
            accounted = binned;
        }
    }
    // Adds the counts of work to the launch's 64-bit totals before 32 bits run
    // over (a single centre can have more than 2^32 pairs).
    __device__ __forceinline__ void report() {
        if (lane == 0) {
            if (tested) atomicAdd(rq.evaluated, (unsigned long long)tested);
            if (binned) atomicAdd(rq.evaluated + 1, (unsigned long long)binned);
        }
        tested = binned = accounted = 0;
    }
    // The centre's triangles: J lists of the near points of view vj, each with
    // K lists of view vk (of one view: with itself, then with the near points
    // after it and the far ones); of two views in both ways round, the second
    // with far points only.  Part (q, kq) of parts x kparts takes the q-th share
    // of J's tiles and the kq-th of K's.
    __device__ __forceinline__ void count(uint32_t centre, int q, int parts, int kq, int kparts) {
        cpos = centre;
        c = J.pts[0][centre];
        const bool self = J.mode & TL_SELF;
        near0 = find_tiles(0);
        near1 = self ? near0 : find_tiles(1);
        if (!near0 || !near1) return;
        for (int pass = 0; pass < (self ? 1 : 2); pass++) {
            const int vj = pass, vk = self ? 0 : 1 - pass;
            const int nt = ntl(vj) <= TL_TILES ? ntl(vj) : J.ntiles[1 + vj];
            const int share = 2 * ((nt + parts - 1) / parts), top = min(2 * nt, (q + 1) * share);
            const int ntk = ntl(vk) <= TL_TILES ? ntl(vk) : J.ntiles[1 + vk];
            const int kshare = 2 * ((ntk + kparts - 1) / kparts), endk = min(2 * ntk, (kq + 1) * kshare);
            int sj = q * share;
            while (sj < top) {
                const int nj = fill(0, vj, TL_NEAR, 0, top, sj);
                if (nj == 0) continue;  // (the steps are used up)
                int sk = kq * kshare, kh = self && kq == 0 ? 0 : 1, nk = nj;
                for (;;) {
                    if (kh && sk >= endk) break;
                    if (kh) nk = fill(1, vk, pass == 0 ? TL_NEAR | TL_FAR : TL_FAR, self ? sj : 0, endk, sk);
                    if (nk > 0) pairs(nj, nk, kh, vj, self ? 1 : vk);
                    if ((tested | binned) >> 31) report();
                    kh = 1;
                }
            }
        }
    }
};

// Persistent; each warp draws items: up to `centres` centres of a job, or one of
// parts x kparts shares of a centre.  The CTA holds the histograms of all `hists`
// output slots of the launch (job: weight >> 32) where they fit; else one, and
// a warp whose item adds to another waits for the others at a CTA barrier,
// where it is flushed.
template <int MODE>
__global__ void __launch_bounds__(TL_MAX_WARPS * 32, 1)
tri_list_kernel(const DevJob* __restrict__ jobs, const uint32_t* __restrict__ item_off, int njobs, unsigned int item0,
                unsigned int nitems, int centres, int parts, int kparts, int hists, unsigned int* counter,
                const __grid_constant__ TriParams p, const __grid_constant__ RecheckQueue rq) {
    extern __shared__ __align__(16) unsigned char smem[];
    TriListWarp* const warps = reinterpret_cast<TriListWarp*>(smem);
    const int nwarps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned int* const H = reinterpret_cast<unsigned int*>(warps + nwarps);
    TriListWarp& W = warps[warp];
    __shared__ unsigned int s_since;  // triangles binned since the last flush
    for (int b = threadIdx.x; b < hists * p.len; b += blockDim.x) H[b] = 0;
    if (threadIdx.x == 0) s_since = 0;
    auto draw = [&]() {
        unsigned int t = 0;
        if (lane == 0) t = atomicAdd(counter, 1u);
        t = __shfl_sync(0xffffffffu, t, 0);
        uint4 it = make_uint4(TASK_NONE, 0, 0, 0);
        if (t < nitems) {
            t += item0;
            const int slot = find_job(item_off, njobs, t);
            const unsigned int l = t - item_off[slot], all = (unsigned)(parts * kparts), first = l / all * centres;
            it = make_uint4((unsigned)slot, first, min((unsigned)centres, (unsigned)jobs[slot].weight - first), l % all);
        }
        __syncwarp();
        if (lane == 0) W.item = it;
        __syncwarp();
    };
    draw();
    unsigned long long* cur = nullptr;
    unsigned long long tested = 0, binned = 0;
    for (;;) {
        __syncthreads();  // every warp waits here with an item for another histogram, or none
        uint32_t next = TASK_NONE;
        for (int q = 0; q < nwarps; q++) next = min(next, warps[q].item.x);  // (TASK_NONE is the largest)
        if (cur && (hists == 1 || next == TASK_NONE)) {
            for (int b = threadIdx.x; b < hists * p.len; b += blockDim.x) {
                const unsigned int v = H[b];
                if (v) {
                    H[b] = 0;
                    atomicAdd((hists == 1 ? cur : rq.hists) + b, (unsigned long long)v);
                }
            }
        }
        if (next == TASK_NONE) break;  // uniform: every thread read the same words
        cur = jobs[next].hist;
        if (threadIdx.x == 0) s_since = 0;
        __syncthreads();
        for (;;) {
            const uint4 it = W.item;
            if (it.x == TASK_NONE || (hists == 1 && jobs[it.x].hist != cur)) break;
            const DevJob& J = jobs[it.x];
            TriCentre<MODE> tc(J, p, W, rq, H, hists, &s_since, it.x);
            for (uint32_t i = 0; i < it.z; i++) tc.count(it.y + i, (int)it.w % parts, parts, (int)it.w / parts, kparts);
            tested += tc.tested;
            binned += tc.binned;
            draw();
        }
    }
    if (lane == 0) {
        if (tested) atomicAdd(rq.evaluated, tested);
        if (binned) atomicAdd(rq.evaluated + 1, binned);
    }
}

cudaError_t launch_tri_list(const DevJob* jobs, const uint32_t* item_off, int njobs, unsigned int item0,
                            unsigned int nitems, int centres, int parts, int kparts, int hists, unsigned int* counter,
                            const TriParams& p, RecheckQueue q, int grid, int warps, int mode, cudaStream_t st) {
    const size_t smem = tri_list_smem_bytes(p.len, hists, warps);
    auto kern = mode == FAST_JBJ ? tri_list_kernel<FAST_JBJ> : mode == FAST_GEOM ? tri_list_kernel<FAST_GEOM>
                                                                                 : tri_list_kernel<FAST_TP>;
    kern<<<grid, warps * 32, smem, st>>>(jobs, item_off, njobs, item0, nitems, centres, parts, kparts, hists, counter, p, q);
    return cudaGetLastError();
}

// JBJ shape parametrization (src/3pcf_C_version_triangle_parametrization_JBJ.cc
// distance(), :116-229): one permutation, s = shortest, q = shortest/middle,
// theta = (longest - middle)/shortest, in float, binned like the triangle
// program; -1 if not counted (zero side, out of range, past the array).
__device__ __forceinline__ int jbj_index(float dist0, float dist1, float dist2, const TriParams& p) {
    float shortest, middle, longest;
    if (dist0 > dist1) {
        if (dist0 > dist2) {
            longest = dist0;
            if (dist1 > dist2) { middle = dist1; shortest = dist2; }
            else { middle = dist2; shortest = dist1; }
        } else {
            middle = dist0;
            if (dist1 > dist2) { longest = dist1; shortest = dist2; }
            else { longest = dist2; shortest = dist1; }
        }
    } else {
        if (dist1 > dist2) {
            longest = dist1;
            if (dist0 > dist2) { middle = dist0; shortest = dist2; }
            else { middle = dist2; shortest = dist0; }
        } else {
            middle = dist1; longest = dist2; shortest = dist0;
        }
    }
    if (dist0 == 0.f || dist1 == 0.f || dist2 == 0.f) return -1;
    const float q = __fdiv_rn(shortest, middle);
    const float th = __fdiv_rn(__fsub_rn(longest, middle), shortest);
    const int i0 = ref_bin_tp<false>(shortest, p.s_lo, p.s_hi, p.S, p.nan_zero);
    const int i1 = ref_bin_tp<false>(q, p.q_lo, p.q_hi, p.Q, p.nan_zero);
    const int i2 = ref_bin_tp<false>(th, p.t_lo, p.t_hi, p.T, p.nan_zero);
    if (i0 < 0 || i1 < 0 || i2 < 0) return -1;
    const long long idx = (long long)p.Q * p.T * i0 + (long long)p.T * i1 + i2;
    return idx < p.len ? (int)idx : -1;
}

// Exact recomputation of queued guard-band triangles (GEOM: of the
// double-precision geometry).
template <int MODE>
__global__ void triangle_recheck_kernel(const DevJob* __restrict__ jobs, RecheckQueue q, TriParams p, AcosTable t) {
    unsigned int n = *q.count;
    if (n > q.cap) n = q.cap;
    for (unsigned int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
        uint4 it = q.items[e];
        const DevJob& J = jobs[it.x & UNIT_SLOT_MASK];
        unsigned w = it.x >> RECHECK_WEIGHT_SHIFT;
        float4 pa = J.pts[0][it.y], pb = J.pts[1][it.z], pc = J.pts[2][it.w];
        if (MODE == FAST_JBJ) {
            const int x = jbj_index(ref_dist<false>(pa, pb), ref_dist<false>(pa, pc), ref_dist<false>(pb, pc), p);
            if (x >= 0) atomicAdd(J.hist + x, (unsigned long long)w);
            continue;
        }
        int out[3];
        if (MODE == FAST_GEOM) tp_geom(geo_dist(pa, pb), geo_dist(pa, pc), geo_dist(pb, pc), p, out);
        else tp_exact<false>(ref_dist<false>(pa, pb), ref_dist<false>(pa, pc), ref_dist<false>(pb, pc), p, t, out);
        for (int k = 0; k < 3; k++)
            if (out[k] >= 0) atomicAdd(J.hist + out[k], (unsigned long long)w);
    }
}

// ---------------------------------------------------------------------------
// Triangle parametrization, plain FP64: every triangle through the exact
// reference arithmetic with each float operation done in FP64.

// Arithmetic of the exact per-triangle kernel.
enum ExactMode : int {
    MODE_FP64 = 0,  // the reference's float arithmetic done in FP64 (identical histograms)
    MODE_GEOM = 1,  // the FP64-geometry truth (tp_geom)
    MODE_JBJ = 2    // the JBJ parametrization in the reference's float arithmetic
};

template <int MODE> struct SideReal { typedef float type; };
template <> struct SideReal<MODE_GEOM> { typedef double type; };

template <int MODE>
__device__ __forceinline__ typename SideReal<MODE>::type side_fp64(float4 a, float4 b) {
    if constexpr (MODE == MODE_GEOM) return geo_dist(a, b);
    else if constexpr (MODE == MODE_JBJ) return ref_dist<false>(a, b);
    else return ref_dist<true>(a, b);
}

template <int PRED, int MODE>
__device__ void triangle_task_fp64(const DevJob& J, uint4 task, int i0, int i1, const TriParams& p, const AcosTable& t,
                                   float4* P, int2* JK, int2* IJ, unsigned int* Hw) {
    typedef typename SideReal<MODE>::type R;  // at most 8 bytes: fits the int2 slots
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const TaskGeom g = task_geom(J, task);
    const bool diag_ij = (J.mode & JOB_B_FROM_A) && task.y == task.z, diag_jk = (J.mode & JOB_C_FROM_B) && task.z == task.w;
    R* jk = reinterpret_cast<R*>(JK);
    load_points(P, J, g);
    __syncthreads();
    for (int e = threadIdx.x; e < TILE * TILE; e += blockDim.x) {
        int j = e / TILE, k = e % TILE;
        if (j < g.nB && k < g.nC) jk[e] = side_fp64<MODE>(P[TILE + j], P[2 * TILE + k]);
    }
    __syncthreads();
    R* row = reinterpret_cast<R*>(IJ + warp * TILE);
    for (int i = i0 + warp; i < min(i1, g.nA); i += TRI_WARPS) {
        const float4 pi = P[i];
        R dik[2];
#pragma unroll
        for (int r = 0; r < 2; r++) {
            int k = lane + 32 * r;
            dik[r] = k < g.nC ? side_fp64<MODE>(pi, P[2 * TILE + k]) : (R)0;
            if (k < g.nB) row[k] = side_fp64<MODE>(pi, P[TILE + k]);
        }
        __syncwarp();
        const int ki = pkey(pi);
        for (int j = diag_ij ? i + 1 : 0; j < g.nB; j++) {
            const R dij = row[j];
            const int kj = pkey(P[TILE + j]);
            if (PRED == PRED_SAME && !(ki <= kj)) continue;
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const int k = lane + 32 * r;
                if (k >= g.nC || (diag_jk && k <= j)) continue;
                unsigned w = 1u;
                const int kkey = pkey(P[2 * TILE + k]);
                if (PRED == PRED_DDR) w = (unsigned)(kkey >= ki) + (unsigned)(kkey >= kj);
                if (PRED == PRED_SAME || PRED == PRED_ONE) w = kj <= kkey ? 1u : 0u;
                if (!w) continue;
                if constexpr (MODE == MODE_JBJ) {
                    const int b = jbj_index(dij, dik[r], jk[j * TILE + k], p);
                    if (b >= 0) atomicAdd(Hw + b, w);
                    continue;
                }
                int out[3];
                if constexpr (MODE == MODE_GEOM) tp_geom(dij, dik[r], jk[j * TILE + k], p, out);
                else tp_exact<true>(dij, dik[r], jk[j * TILE + k], p, t, out);
                for (int b = 0; b < 3; b++)
                    if (out[b] >= 0) atomicAdd(Hw + out[b], w);
            }
        }
        __syncwarp();
    }
}

template <int MODE>
__global__ void __launch_bounds__(TRI_THREADS, 1)
triangle_fp64_kernel(const DevJob* __restrict__ jobs, UnitList ul, unsigned int* counter, TriParams p, AcosTable t,
                     int copies) {
    extern __shared__ __align__(16) unsigned char smem[];
    float4* P = reinterpret_cast<float4*>(smem);
    int2* JK = reinterpret_cast<int2*>(smem + 3 * TILE * sizeof(float4));
    int2* IJ = JK + TILE * TILE;
    unsigned int* H = reinterpret_cast<unsigned int*>(IJ + TRI_WARPS * TILE);
    __shared__ uint4 s_task;
    __shared__ int s_i0, s_i1;
    for (int b = threadIdx.x; b < copies * p.len; b += blockDim.x) H[b] = 0;
    unsigned int* Hw = H + ((threadIdx.x >> 5) % copies) * p.len;
    int cur = -1;
    unsigned int since = 0;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) s_task = draw_unit(ul, counter, s_i0, s_i1);
        __syncthreads();
        const uint4 task = s_task;
        const int slot = task.x == TASK_NONE ? -1 : (int)task.x;
        if ((slot != cur || since >= FLUSH_EVERY) && cur >= 0) {
            flush_hist(H, copies, p.len, jobs[cur].hist);
            since = 0;
        }
        cur = slot;
        if (slot < 0) break;
        since++;
        const DevJob& J = jobs[slot];
        switch (J.mode & JOB_PRED_MASK) {
            case PRED_NONE: triangle_task_fp64<PRED_NONE, MODE>(J, task, s_i0, s_i1, p, t, P, JK, IJ, Hw); break;
            case PRED_DDR: triangle_task_fp64<PRED_DDR, MODE>(J, task, s_i0, s_i1, p, t, P, JK, IJ, Hw); break;
            case PRED_SAME: triangle_task_fp64<PRED_SAME, MODE>(J, task, s_i0, s_i1, p, t, P, JK, IJ, Hw); break;
            default: triangle_task_fp64<PRED_ONE, MODE>(J, task, s_i0, s_i1, p, t, P, JK, IJ, Hw); break;
        }
    }
}

// ---------------------------------------------------------------------------
// Three-side histogram (src/3pcf_C_version.cc): every ordered triple, sides in
// source order d01 -> i0, d02 -> i1, d12 -> i2, index n^2 i2 + n i1 + i0.

constexpr int TS_WARPS = 8;  // warps per CTA, or per group of the grouped kernel
constexpr int TS_GROUP_THREADS = TS_WARPS * 32;
constexpr int TS_GROUPS_MAX = 4;
constexpr uint32_t TS_FAR = 1u << 30;
// A copy receives at most 64^3 = 2^18 counts per task, so 8192 tasks keep
// every 32-bit shared counter below 2^31.
constexpr unsigned int TS_FLUSH_EVERY = 8192;

// Per warp: the i-k and i-j code rows of its point i and a queue of (j, k)
// candidates (up to 31 left over plus 64 from one j).
constexpr int TS_QCAP = 96;
constexpr int TS_ROW = 2 * TILE + TS_QCAP;

// Shared memory of one task pipeline (an 8-warp CTA, or one group of the
// grouped kernel): point tiles, j-k table, per-warp rows, j-k masks, boxes,
// next point.  The j-k table holds 32-bit codes; in clean mode it holds the
// bins alone (only sides below hist_max are ever read), one byte each up to
// 255 bins.
struct TsLayout {
    size_t jk, rows, jkm, box, flags, next, bytes;
};
__host__ __device__ constexpr bool ts_byte_jk(const ThreeParams& p) { return p.clean && p.n <= 255; }
__host__ __device__ constexpr TsLayout ts_layout(bool byte_jk) {
    const size_t jk = 3 * TILE * sizeof(float4);
    const size_t rows = jk + (byte_jk ? TILE * TILE : TILE * TILE * sizeof(uint32_t));
    const size_t jkm = rows + TS_WARPS * TS_ROW * sizeof(uint32_t);
    const size_t box = jkm + TILE * sizeof(unsigned long long);
    const size_t flags = box + 36 * sizeof(float);  // reach flags of the points of tiles B and A
    const size_t next = flags + 2 * TILE;
    return TsLayout{jk, rows, jkm, box, flags, next, (next + sizeof(int) + 127) & ~(size_t)127};
}

// distance_to_bin of src/3pcf_C_version.cc:23-51, times 'scale'; sides at or
// above hist_max give nbins+1 (reference) or, in clean mode, a value that
// pushes every derived index out of range.
template <bool FP64>
__device__ __forceinline__ uint32_t side_code3(float d, const ThreeParams& p, uint32_t scale) {
    typedef FOps<FP64> F;
    if (d < p.lo) return 0u;
    if (d >= p.hi) return p.clean ? TS_FAR : (uint32_t)(p.n + 1) * scale;
    return (uint32_t)__float2int_rz(F::div(F::sub(d, p.lo), p.bw)) * scale;
}

// Three-side code of the side a-b.  The guarded FP32 kernel skips the square
// root and the division: the bin is a non-decreasing step function of the
// squared length, so a first guess from an approximate square root (within one
// bin) is corrected against the exact thresholds U of the two neighbouring
// steps.  The plain FP64 kernel evaluates the reference's formula.
template <bool FP64>
__device__ __forceinline__ uint32_t side_code3_pts(float4 a, float4 b, const ThreeParams& p, const float* U,
                                                   uint32_t scale) {
    if (!FP64 && p.fast) {
        const float dx = __fsub_rn(a.x, b.x), dy = __fsub_rn(a.y, b.y), dz = __fsub_rn(a.z, b.z);
        float d2 = __fmul_rn(dx, dx);
        d2 = __fadd_rn(d2, __fmul_rn(dy, dy));
        d2 = __fadd_rn(d2, __fmul_rn(dz, dz));
        float da;
        asm("sqrt.approx.f32 %0, %1;" : "=f"(da) : "f"(d2));
        // the guess rounds to nearest: where d reaches hi the code jumps over
        // nbins (unless rounding gives bin nbins), and a truncated guess just
        // below hi would be two steps short
        int v = __float2int_rn(__fmul_rn(__fsub_rn(da, p.lo), p.inv_bw));
        v = min(max(v, 0), p.n + 1);
        v = v - 1 + (d2 >= U[v] ? 1 : 0) + (d2 >= U[v + 1] ? 1 : 0);
        if (v > p.n) return p.clean ? TS_FAR : (uint32_t)(p.n + 1) * scale;
        return (uint32_t)v * scale;
    }
    return side_code3<FP64>(ref_dist<FP64>(a, b), p, scale);
}

// Symmetric three-side tasks (one catalog in all roles) visit each multiset
// {i <= j <= k} once.  With a shared histogram they count it once in a
// multiset accumulator (m = nbins + 2 codes per side, so no index aliases):
//   U[v_jk m^2 + v_ik m + v_ij]   three distinct points,
//   U2[v]                         two equal indices (sides 0, v, v),
//   U6                            i == j == k,
// which ts_flush expands into the reference's ordered histogram.  The
// accumulator is ts_acc_words(p) words, U2 from word ts_u2(p).
__host__ __device__ inline int ts_u2(const ThreeParams& p) {
    const int m = p.n + 2;
    return hist_stride(m * m * m);
}
__host__ __device__ inline int ts_acc_words(const ThreeParams& p) {
    const int acc = ts_u2(p) + p.n + 3;
    return acc > p.len ? acc : p.len;
}

// Adds one ordering (sides d01, d02, d12 with codes x0, x1, x2) of a triple
// to the reference's histogram (an index at or past its end is dropped).
__device__ __forceinline__ void ts_put(unsigned long long* g, uint32_t x0, uint32_t x1, uint32_t x2,
                                       const ThreeParams& p, unsigned long long u) {
    const uint32_t t = x2 * (uint32_t)p.n * (uint32_t)p.n + x1 * (uint32_t)p.n + x0;
    if (t < (uint32_t)p.len) atomicAdd(g + t, u);
}

// The distinct orderings of a multiset with side codes (v_ij, v_ik, v_jk):
// (i,j,k) (ij,ik,jk), (i,k,j) (ik,ij,jk), (j,i,k) (ij,jk,ik), (j,k,i) (jk,ij,ik),
// (k,i,j) (ik,jk,ij), (k,j,i) (jk,ik,ij); with i == j or j == k three of them.
__device__ __forceinline__ void ts_put_orderings(unsigned long long* g, uint32_t vij, uint32_t vik, uint32_t vjk,
                                                 bool eij, bool ejk, const ThreeParams& p, unsigned long long u) {
    ts_put(g, vij, vik, vjk, p, u);
    if (!ejk) ts_put(g, vik, vij, vjk, p, u);
    if (!eij) ts_put(g, vij, vjk, vik, p, u);
    if (!eij) ts_put(g, vjk, vij, vik, p, u);
    if (!ejk) ts_put(g, vik, vjk, vij, p, u);
    if (!eij && !ejk) ts_put(g, vjk, vik, vij, p, u);
}

// Flushes 'copies' shared copies (hist_stride(ts_acc_words(p)) words apart)
// into the job's 64-bit histogram: the swizzled ordered histogram, or the
// multiset accumulator of a symmetric job expanded into its orderings.
__device__ void ts_flush(unsigned int* H, int copies, const ThreeParams& p, unsigned long long* g, bool sym) {
    const int stride = hist_stride(ts_acc_words(p));
    __syncthreads();
    if (!sym) {
        for (int b = threadIdx.x; b < p.len; b += blockDim.x) {
            const int at = (int)hist_pos((unsigned)b);
            unsigned long long u = 0;
            for (int c = 0; c < copies; c++) {
                u += H[c * stride + at];
                H[c * stride + at] = 0;
            }
            if (u) atomicAdd(g + b, u);
        }
    } else {
        const int m = p.n + 2, m3 = m * m * m, u2 = ts_u2(p);
        const uint32_t z = (uint32_t)p.zcode;
        for (int b = threadIdx.x; b < m3 + m + 1; b += blockDim.x) {
            const int at = b < m3 ? (int)hist_pos((unsigned)b) : u2 + (b - m3);
            unsigned long long u = 0;
            for (int c = 0; c < copies; c++) {
                u += H[c * stride + at];
                H[c * stride + at] = 0;
            }
            if (!u) continue;
            if (b < m3) {
                const uint32_t vij = b % m, vik = (b / m) % m, vjk = b / (m * m);
                ts_put_orderings(g, vij, vik, vjk, false, false, p, u);
            } else if (b < m3 + m) {
                const uint32_t v = b - m3;  // (i, i, k) or (i, k, k): sides 0, v, v
                ts_put(g, z, v, v, p, u);
                ts_put(g, v, z, v, p, u);
                ts_put(g, v, v, z, p, u);
            } else {
                ts_put(g, z, z, z, p, u);
            }
        }
    }
    __syncthreads();
}

// One task pipeline: its threads (tid in [0, 256)), and its barrier (0: the
// CTA's, else a named barrier of its 256 threads).
struct TsPipe {
    int tid, warp, lane, bar;
    __device__ __forceinline__ void sync() const {
        if (bar == 0) __syncthreads();
        else asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(TS_GROUP_THREADS) : "memory");
    }
};

// Bounding boxes of the three tiles (two 32-point halves each) into BX, one
// warp per half; the caller synchronises.
__device__ __forceinline__ void tile_boxes(const float4* P, const TaskGeom& g, float* BX, int warp, int lane) {
    if (warp >= 6) return;
    const int role = warp >> 1, idx = (warp & 1) * 32 + lane;
    const int n = role == 0 ? g.nA : (role == 1 ? g.nB : g.nC);
    const float4 pt = P[role * TILE + idx];
    const bool valid = idx < n;
    float lo[3] = {valid ? pt.x : INFINITY, valid ? pt.y : INFINITY, valid ? pt.z : INFINITY};
    float hi[3] = {valid ? pt.x : -INFINITY, valid ? pt.y : -INFINITY, valid ? pt.z : -INFINITY};
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int a = 0; a < 3; a++) {
            lo[a] = fminf(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], o));
            hi[a] = fmaxf(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], o));
        }
    if (lane == 0) {
#pragma unroll
        for (int a = 0; a < 3; a++) {
            BX[warp * 6 + a] = lo[a];
            BX[warp * 6 + 3 + a] = hi[a];
        }
    }
}

// True if every point of half-tile box 'b' (role * 2 + half) is at least
// 'reach' from pt; an empty half (inverted box) is far from everything.
__device__ __forceinline__ bool far_from_box(const float* BX, float4 pt, int b, float reach2) {
    const float* b0 = BX + b * 6;
    const float gx = fmaxf(0.f, fmaxf(b0[0] - pt.x, pt.x - b0[3]));
    const float gy = fmaxf(0.f, fmaxf(b0[1] - pt.y, pt.y - b0[4]));
    const float gz = fmaxf(0.f, fmaxf(b0[2] - pt.z, pt.z - b0[5]));
    return fmaf(gz, gz, fmaf(gy, gy, gx * gx)) >= reach2;
}

// One task (tiles A, B, C) of the three-side histogram on one pipeline whose
// shared memory starts at 'base'; counts go to the shared copy Hw (swizzled)
// or, with GLOBAL_HIST, straight to the job's 64-bit histogram.
template <bool FP64, bool GLOBAL_HIST>
__device__ void three_side_task(const DevJob& J, uint4 task, int i0, int i1, const ThreeParams& p, const float* U,
                                unsigned char* base, unsigned int* Hw, const TsPipe& pp) {
    float4* P = reinterpret_cast<float4*>(base);
    const bool byte_jk = ts_byte_jk(p);
    const TsLayout L = ts_layout(byte_jk);
    uint8_t* FJ = base + L.flags;  // per j of tile B: 1 reaches tile A, 2 / 4 reaches half 0 / 1 of tile C
    uint8_t* FI = FJ + TILE;       // per i of tile A: 1 / 2 reaches half 0 / 1 of B, 4 / 8 of C
    uint32_t* JK = reinterpret_cast<uint32_t*>(base + L.jk);
    uint8_t* JK8 = base + L.jk;
    uint32_t* ROWS = reinterpret_cast<uint32_t*>(base + L.rows);
    unsigned long long* JKM = reinterpret_cast<unsigned long long*>(base + L.jkm);
    float* BX = reinterpret_cast<float*>(base + L.box);
    int* next_i = reinterpret_cast<int*>(base + L.next);
    const int warp = pp.warp, lane = pp.lane;
    const TaskGeom g = task_geom(J, task);
    const uint32_t n = p.n, n2 = (uint32_t)p.n * p.n, len = (uint32_t)p.len;
    const uint32_t m = n + 2, mm = m * m, u2 = (uint32_t)ts_u2(p);  // multiset accumulator
    // Symmetric tasks (one catalog in all three roles): tiles a <= b <= c and,
    // on diagonal tile pairs, positions i <= j <= k, so that every multiset
    // {i, j, k} is visited once and counted for all its orderings.
    const bool sym = (J.mode & JOB_PRED_MASK) == PRED_SAME;
    const bool diag_ij = (J.mode & JOB_B_FROM_A) && task.y == task.z, diag_jk = (J.mode & JOB_C_FROM_B) && task.z == task.w;
    i1 = min(i1, g.nA);  // the unit's points of tile A
    for (int t = pp.tid; t < 3 * TILE; t += TS_GROUP_THREADS) {
        const int role = t / TILE, idx = t % TILE;
        const int nr = role == 0 ? g.nA : (role == 1 ? g.nB : g.nC);
        const int b0 = role == 0 ? g.a0 : (role == 1 ? g.b0 : g.c0);
        P[t] = idx < nr ? J.pts[role][b0 + idx] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (pp.tid == 0) *next_i = i0;
    pp.sync();
    if (p.clean) {
        // Clean mode drops every triple with a side >= hist_max, so a point
        // farther than that from a whole tile takes no part in the task (the
        // 1e-5 margin covers the rounding of the bound and of the distance).
        tile_boxes(P, g, BX, warp, lane);
        pp.sync();
        const float reach = p.hi * (1.0f + 1e-5f), reach2 = reach * reach;
        // reach flags of every point against the half-tile boxes, lane-parallel
        if (warp == 0) {
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const int j = lane + 32 * r;
                const float4 pj = P[TILE + j];
                unsigned f = 0;
                if (!far_from_box(BX, pj, 0, reach2) || !far_from_box(BX, pj, 1, reach2)) f |= 1u;
                if (!far_from_box(BX, pj, 4, reach2)) f |= 2u;
                if (!far_from_box(BX, pj, 5, reach2)) f |= 4u;
                FJ[j] = (uint8_t)f;
            }
        } else if (warp == 1) {
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const int i = lane + 32 * r;
                const float4 pi = P[i];
                unsigned f = 0;
                if (!far_from_box(BX, pi, 2, reach2)) f |= 1u;
                if (!far_from_box(BX, pi, 3, reach2)) f |= 2u;
                if (!far_from_box(BX, pi, 4, reach2)) f |= 4u;
                if (!far_from_box(BX, pi, 5, reach2)) f |= 8u;
                FI[i] = (uint8_t)f;
            }
        }
        pp.sync();
        // j-k codes, one warp per row j, and JKM[j]: the k's whose side is
        // below hist_max (halves of tile C out of reach of j are skipped)
        for (int j = warp; j < g.nB; j += TS_WARPS) {
            const float4 pj = P[TILE + j];
            const unsigned f = FJ[j];
            if (!(f & 1u) || !(f & 6u)) {  // no i, or no k, reaches j: the row is never read
                if (lane == 0) JKM[j] = 0ull;
                continue;
            }
            uint32_t c0 = TS_FAR, c1 = TS_FAR;
            if ((f & 2u) && lane < g.nC) c0 = side_code3_pts<FP64>(pj, P[2 * TILE + lane], p, U, 1u);
            if ((f & 4u) && lane + 32 < g.nC) c1 = side_code3_pts<FP64>(pj, P[2 * TILE + lane + 32], p, U, 1u);
            if (byte_jk) {  // bins <= nbins <= 255 where read
                JK8[j * TILE + lane] = (uint8_t)c0;
                JK8[j * TILE + lane + 32] = (uint8_t)c1;
            } else {
                JK[j * TILE + lane] = c0;
                JK[j * TILE + lane + 32] = c1;
            }
            unsigned long long m = ballot64(c0 < TS_FAR, c1 < TS_FAR);
            if (sym && diag_jk) m &= ~0ull << j;  // k >= j
            if (lane == 0) JKM[j] = m;
        }
        pp.sync();
        uint32_t* row_ik = ROWS + warp * TS_ROW;
        uint32_t* row_ij = row_ik + TILE;
        uint32_t* cq = row_ij + TILE;
        const unsigned lt = (1u << lane) - 1u;
        auto add = [&](uint32_t idx) {
            if (idx < len) {  // a side rounded to bin nbins aliases as in the reference
                if (GLOBAL_HIST) atomicAdd(J.hist + idx, 1ull);
                else atomicAdd(Hw + hist_pos(idx), 1u);
            }
        };
        int i = 0;
        auto count_candidates = [&](const uint32_t* e, int cnt) {
            if (lane < cnt) {
                const uint32_t c = e[lane];
                const int j = c & 63, k = c >> 6;
                const uint32_t vjk = byte_jk ? (uint32_t)JK8[j * TILE + k] : JK[j * TILE + k];
                const uint32_t vik = row_ik[k], vij = row_ij[j];
                if (!sym) {
                    add(vjk * n2 + vik * n + vij);
                } else {
                    const bool eij = diag_ij && i == j, ejk = diag_jk && j == k;
                    if (GLOBAL_HIST) ts_put_orderings(J.hist, vij, vik, vjk, eij, ejk, p, 1ull);
                    else if (!eij && !ejk) atomicAdd(Hw + hist_pos(vjk * mm + vik * m + vij), 1u);
                    else atomicAdd(Hw + u2 + (eij && ejk ? m : (eij ? vik : vij)), 1u);
                }
            }
        };
        for (;;) {
            // points of tile A go to warps one at a time (their work is uneven)
            i = 0;
            if (lane == 0) i = atomicAdd(next_i, 1);
            i = __shfl_sync(0xffffffffu, i, 0);
            if (i >= i1) break;
            const float4 pi = P[i];
            const unsigned fi = FI[i];
            if (!(fi & 3u) || !(fi & 12u)) continue;  // out of reach of tile B or tile C (warp-uniform)
            uint32_t cik[2], cij[2];
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const int k = lane + 32 * r;
                cik[r] = ((fi >> (2 + r)) & 1u) && k < g.nC ? side_code3_pts<FP64>(pi, P[2 * TILE + k], p, U, 1u)
                                                             : TS_FAR;
            }
            const unsigned long long mk = ballot64(cik[0] < TS_FAR, cik[1] < TS_FAR);
            if (!mk) continue;  // warp-uniform
            // j's with a usable i-j side and a k usable with both i and j
            bool vj[2];
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const int j = lane + 32 * r;
                cij[r] = TS_FAR;
                vj[r] = false;
                if (((fi >> r) & 1u) && j < g.nB && (JKM[j] & mk) && !(sym && diag_ij && j < i)) {
                    cij[r] = side_code3_pts<FP64>(pi, P[TILE + j], p, U, 1u);
                    vj[r] = cij[r] < TS_FAR;
                }
            }
            unsigned long long mj = ballot64(vj[0], vj[1]);
            // Candidates (j, k) of this i, every j in turn, queued by the
            // whole warp and counted 32 at a time.
            row_ik[lane] = cik[0];
            row_ik[lane + 32] = cik[1];
            row_ij[lane] = cij[0];
            row_ij[lane + 32] = cij[1];
            int qn = 0;  // warp-uniform
            while (mj) {
                const int j = __ffsll((long long)mj) - 1;
                mj &= mj - 1ull;
                const unsigned long long cm = mk & JKM[j];
                const unsigned lo = (unsigned)cm, hi = (unsigned)(cm >> 32);
                const int nlo = __popc(lo);
                if ((lo >> lane) & 1u) cq[qn + __popc(lo & lt)] = (uint32_t)j | ((uint32_t)lane << 6);
                if ((hi >> lane) & 1u) cq[qn + nlo + __popc(hi & lt)] = (uint32_t)j | ((uint32_t)(lane + 32) << 6);
                qn += nlo + __popc(hi);
                __syncwarp();
                while (qn >= 32) {
                    qn -= 32;
                    count_candidates(cq + qn, 32);
                    __syncwarp();
                }
            }
            if (qn > 0) count_candidates(cq, qn);
            __syncwarp();
        }
        return;
    }
    if (sym) {
        // every multiset {i <= j <= k} of the task (codes 0 .. nbins + 1)
        for (int e = pp.tid; e < TILE * TILE; e += TS_GROUP_THREADS) {
            const int j = e / TILE, k = e % TILE;
            JK[e] = (j < g.nB && k < g.nC) ? side_code3_pts<FP64>(P[TILE + j], P[2 * TILE + k], p, U, 1u) : 0u;
        }
        pp.sync();
        uint32_t* row = ROWS + warp * TS_ROW;
        for (int i = i0 + warp; i < i1; i += TS_WARPS) {
            const float4 pi = P[i];
            uint32_t vik[2];
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const int k = lane + 32 * r;
                vik[r] = k < g.nC ? side_code3_pts<FP64>(pi, P[2 * TILE + k], p, U, 1u) : 0u;
                if (lane + 32 * r < g.nB) row[lane + 32 * r] = side_code3_pts<FP64>(pi, P[TILE + lane + 32 * r], p, U, 1u);
            }
            __syncwarp();
            if (!GLOBAL_HIST && !diag_ij && !diag_jk) {
                // three tiles apart: every (j, k) is a multiset of distinct points
                const uint32_t vikm0 = vik[0] * m, vikm1 = vik[1] * m;
                const bool k0 = lane < g.nC, k1 = lane + 32 < g.nC;
#pragma unroll 4
                for (int j = 0; j < g.nB; j++) {
                    const uint32_t vij = row[j];
                    if (k0) atomicAdd(Hw + hist_pos(JK[j * TILE + lane] * mm + vikm0 + vij), 1u);
                    if (k1) atomicAdd(Hw + hist_pos(JK[j * TILE + lane + 32] * mm + vikm1 + vij), 1u);
                }
                __syncwarp();
                continue;
            }
            for (int j = diag_ij ? i : 0; j < g.nB; j++) {
                const uint32_t vij = row[j];
                const bool eij = diag_ij && j == i;
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    const int k = lane + 32 * r;
                    if (k >= g.nC || (diag_jk && k < j)) continue;
                    const bool ejk = diag_jk && k == j;
                    const uint32_t vjk = JK[j * TILE + k];
                    if (GLOBAL_HIST) ts_put_orderings(J.hist, vij, vik[r], vjk, eij, ejk, p, 1ull);
                    else if (!eij && !ejk) atomicAdd(Hw + hist_pos(vjk * mm + vik[r] * m + vij), 1u);
                    else atomicAdd(Hw + u2 + (eij && ejk ? m : (eij ? vik[r] : vij)), 1u);
                }
            }
            __syncwarp();
        }
        return;
    }
    for (int e = pp.tid; e < TILE * TILE; e += TS_GROUP_THREADS) {
        const int j = e / TILE, k = e % TILE;
        JK[e] = (j < g.nB && k < g.nC) ? side_code3_pts<FP64>(P[TILE + j], P[2 * TILE + k], p, U, n2)
                                       : TS_FAR;
    }
    pp.sync();
    uint32_t* row = ROWS + warp * TS_ROW;
    for (int i = i0 + warp; i < i1; i += TS_WARPS) {
        const float4 pi = P[i];
        uint32_t cik[2];
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const int k = lane + 32 * r;
            cik[r] = k < g.nC ? side_code3_pts<FP64>(pi, P[2 * TILE + k], p, U, n) : TS_FAR;
        }
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const int k = lane + 32 * r;
            if (k < g.nB) row[k] = side_code3_pts<FP64>(pi, P[TILE + k], p, U, 1u);
        }
        __syncwarp();
#pragma unroll 4
        for (int j = 0; j < g.nB; j++) {
            const uint32_t cij = row[j];
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const int k = lane + 32 * r;
                const uint32_t idx = JK[j * TILE + k] + cik[r] + cij;
                if (idx < len) {
                    if (GLOBAL_HIST) atomicAdd(J.hist + idx, 1ull);
                    else atomicAdd(Hw + hist_pos(idx), 1u);
                }
            }
        }
        __syncwarp();
    }
}

// 8-warp CTAs, several per SM: warp-private shared histogram copies (copies
// > 0) or the global histogram.
template <bool FP64, bool GLOBAL_HIST>
__global__ void __launch_bounds__(TS_GROUP_THREADS, 4)
three_side_kernel(const DevJob* __restrict__ jobs, UnitList ul, unsigned int* counter, ThreeParams p, int copies) {
    extern __shared__ __align__(16) unsigned char smem[];
    unsigned int* H = reinterpret_cast<unsigned int*>(smem + ts_layout(ts_byte_jk(p)).bytes);
    __shared__ uint4 s_task;
    __shared__ int s_i0, s_i1;
    __shared__ float s_u[TS_UMAX];
    for (int v = threadIdx.x; v < TS_UMAX; v += blockDim.x) s_u[v] = p.u[v];
    const int stride = hist_stride(ts_acc_words(p));
    if (!GLOBAL_HIST)
        for (int b = threadIdx.x; b < copies * stride; b += blockDim.x) H[b] = 0;
    unsigned int* Hw = H + (GLOBAL_HIST ? 0 : ((threadIdx.x >> 5) % copies) * stride);
    bool cur_sym = false;
    const TsPipe pp{(int)threadIdx.x, (int)(threadIdx.x >> 5), (int)(threadIdx.x & 31), 0};
    int cur = -1;
    unsigned int since = 0;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) s_task = draw_unit(ul, counter, s_i0, s_i1);
        __syncthreads();
        const uint4 task = s_task;
        const int slot = task.x == TASK_NONE ? -1 : (int)task.x;
        if (!GLOBAL_HIST && (slot != cur || since >= TS_FLUSH_EVERY) && cur >= 0) {
            ts_flush(H, copies, p, jobs[cur].hist, cur_sym);
            since = 0;
        }
        cur = slot;
        if (slot < 0) break;
        cur_sym = (jobs[slot].mode & JOB_PRED_MASK) == PRED_SAME;
        since++;
        three_side_task<FP64, GLOBAL_HIST>(jobs[slot], task, s_i0, s_i1, p, s_u, smem, Hw, pp);
    }
}

// One CTA per SM of 'groups' independent 8-warp task pipelines (named
// barriers 1..groups) around one shared histogram too large for several
// CTAs per SM.  A pipeline runs tasks of the current job until it draws a
// task of another job (or none), or the CTA has run TS_FLUSH_EVERY tasks since
// the last flush; then it waits for the others at a CTA barrier, where the
// histogram is flushed and the next current job is the smallest one held.
// Every pipeline reaches that barrier: each runs finitely many tasks of the
// current job.  At most TS_FLUSH_EVERY + groups - 1 tasks are counted between
// two flushes, each at most 2^18 per bin, so the 32-bit counters cannot wrap.
template <bool FP64>
__global__ void __launch_bounds__(TS_GROUPS_MAX * TS_GROUP_THREADS, 1)
three_side_grouped_kernel(const DevJob* __restrict__ jobs, UnitList ul, unsigned int* counter, ThreeParams p,
                          int groups) {
    extern __shared__ __align__(16) unsigned char smem[];
    const size_t pipe_bytes = ts_layout(ts_byte_jk(p)).bytes;
    unsigned int* H = reinterpret_cast<unsigned int*>(smem + (size_t)groups * pipe_bytes);
    __shared__ uint4 s_task[TS_GROUPS_MAX];
    __shared__ int2 s_i[TS_GROUPS_MAX];  // its points of tile A
    __shared__ unsigned int s_stop[TS_GROUPS_MAX];  // the pipeline leaves the job to flush
    __shared__ unsigned int s_since;                // tasks run since the last flush
    __shared__ float s_u[TS_UMAX];
    for (int v = threadIdx.x; v < TS_UMAX; v += blockDim.x) s_u[v] = p.u[v];
    const int gi = threadIdx.x / TS_GROUP_THREADS, gt = threadIdx.x % TS_GROUP_THREADS;
    const TsPipe pp{gt, gt >> 5, gt & 31, 1 + gi};
    unsigned char* base = smem + (size_t)gi * pipe_bytes;
    for (int b = threadIdx.x; b < hist_stride(ts_acc_words(p)); b += blockDim.x) H[b] = 0;
    if (threadIdx.x == 0) s_since = 0;
    auto draw = [&]() {
        if (gt == 0) s_task[gi] = draw_unit(ul, counter, s_i[gi].x, s_i[gi].y);
    };
    draw();
    int cur = -1;
    bool cur_sym = false;
    for (;;) {
        __syncthreads();  // every pipeline waits here with a task of another job, or none
        if (cur >= 0) ts_flush(H, 1, p, jobs[cur].hist, cur_sym);
        uint32_t next = TASK_NONE;
        for (int g2 = 0; g2 < groups; g2++) {
            const uint32_t x = s_task[g2].x;
            if (x != TASK_NONE) next = min(next, x);
        }
        if (next == TASK_NONE) break;  // uniform: every thread read the same words
        cur_sym = (jobs[next].mode & JOB_PRED_MASK) == PRED_SAME;
        if (threadIdx.x < TS_GROUPS_MAX) s_stop[threadIdx.x] = 0;
        if (threadIdx.x == 0) s_since = 0;
        __syncthreads();
        cur = (int)next;
        for (;;) {
            // s_task[gi] and s_stop[gi] change only between this pipeline's barriers
            const uint4 task = s_task[gi];
            if (task.x == TASK_NONE || (int)task.x != cur || s_stop[gi]) break;
            three_side_task<FP64, false>(jobs[cur], task, s_i[gi].x, s_i[gi].y, p, s_u, base, H, pp);
            pp.sync();  // the pipeline is done with s_task[gi] and its buffers
            if (gt == 0) s_stop[gi] = atomicAdd(&s_since, 1u) + 1 >= TS_FLUSH_EVERY;
            draw();
            pp.sync();
        }
    }
}

// Squared gap of two tile boxes (reduced by a margin that covers the rounding
// of the bound and of the reference's separation) below reach2: the tiles can
// hold a counted pair.
__device__ __forceinline__ bool boxes_near(const float4* __restrict__ A, const float4* __restrict__ B, float reach2) {
    const float4 al = A[0], ah = A[1], bl = B[0], bh = B[1];
    const float gx = fmaxf(0.f, fmaxf(al.x - bh.x, bl.x - ah.x));
    const float gy = fmaxf(0.f, fmaxf(al.y - bh.y, bl.y - ah.y));
    const float gz = fmaxf(0.f, fmaxf(al.z - bh.z, bl.z - ah.z));
    // (an overflowing gap is kept below an infinite reach only)
    return !((gx * gx + gy * gy + gz * gz) * (1.0f - 4e-5f) >= reach2);
}

// ---------------------------------------------------------------------------
// Three-side histogram from neighbour lists.
//
// Only triples with all three sides below hist_max are enumerated: for each
// point of the centre role, the points of the other two roles below hist_max
// from it go into a list in shared memory (coordinates and four times the side
// code), and
// every pair of the list gets its third side.  The reference's mode also
// counts triples with sides at or above hist_max (code F = n + 1); an index
// with F in its last place (n^2 F > n^3) is past the array's end, and the rest
// follow from the near triples T and from pairs of near sides at one point:
//   T(a,F,c) = WB(a,c) - sum_b T(a,b,c),  WB(a,c) = sum over j of hA_j(a) hC_j(c)
//   T(F,b,c) = WC(b,c) - sum_a T(a,b,c),  WC(b,c) = sum over k of hA_k(b) hB_k(c)
//   T(F,F,c) = nA PBC(c) - sum_ab T(a,b,c) - sum_a T(a,F,c) - sum_b T(F,b,c)
// with hX_p(v) the number of points of role X at code v from p and PBC the
// pairs of B and C at code c.  All linear in counts, so near counts and the
// sums W and P are collected per accumulator (three_near_kernel,
// three_wedge_kernel) and expanded once (three_expand_kernel).
//
// Bound by the issue rate and the shared-memory atomics of the pairs of the
// lists.  (Against tiles of 64^3 triples with class masks, whose rows and
// candidate queues were most of the work: 150k lattice points, 32 bins,
// 25.8 ms; D-D-D to R-R-R of 3k points, 16 bins, 23.4 ms.)

constexpr int NEAR_CAP = 1024;        // list entries of a pipeline (halves of 512 for two lists)
constexpr int NEAR_TILES = 256;       // near tiles of a centre's tile, per list
constexpr int NEAR_CHUNK = 8;         // tiles of a half list where the lists overflow
constexpr int NEAR_MAX_POINTS = NEAR_TILES * TILE;
constexpr float NEAR_PAD = 1e18f;     // coordinate of padding entries: out of every range

struct NearPipe {
    float x[NEAR_CAP], y[NEAR_CAP], z[NEAR_CAP];
    uint32_t code[NEAR_CAP];
    uint32_t tiles[2][NEAR_TILES];
    int ntiles[2], count[2];
    uint4 item;  // job, tile, first centre, (unused)
    unsigned int stop;
};

// Accumulator words (64 bits each): near triples, two equal indices, three
// equal, then the wedges and pairs.
__host__ __device__ inline int near_words3(int n) { return (n + 1) * (n + 1) * (n + 1); }
size_t three_near_acc_words(int n) {
    const size_t m = n + 1;
    return m * m * m + m + 1 + 2 * m * m + m;
}
// Shared words of the near triples: strides that spread the banks (odd, and
// different modulo 32), then the codes of two equal indices, then one word.
struct NearStride {
    int q, r, u2, words;
};
__host__ __device__ inline NearStride near_stride(int n) {
    NearStride s;
    const int m = n + 1;
    s.q = m | 1;
    s.r = (m * s.q) | 1;
    if ((s.r & 31) == (s.q & 31)) s.r += 2;
    s.u2 = m * s.r;
    s.words = (s.u2 + m + 1 + 31) & ~31;
    return s;
}
size_t three_near_smem_bytes(int n, int pipes) { return (size_t)pipes * sizeof(NearPipe) + (size_t)near_stride(n).words * 4; }

// Exact three-side code, or -1 at or above hist_max.
__device__ __forceinline__ int near_exact(float4 a, float4 b, const NearParams& p) {
    const float d = ref_dist<false>(a, b);
    if (d < p.lo) return 0;
    if (d >= p.hi) return -1;
    return __float2int_rz(__fdiv_rn(__fsub_rn(d, p.lo), p.bw));
}

// The same from rsqrt.approx outside the guard band (see pair_guard).
__device__ __forceinline__ int near_code(float4 a, float4 b, const NearParams& p) {
    const float dx = a.x - b.x, dy = a.y - b.y, dz = a.z - b.z;
    const float d2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
    const GuardedBin g = magic_floor(fmaf(d2 * rsqrt_approx(d2), p.inv_bw, p.off));
    if (!(fabsf(g.err) <= p.thr)) return near_exact(a, b, p);
    return g.bin < p.n ? max(g.bin, 0) : -1;
}

// Every pair (entry j of [j0, j1), this lane's entry k) of two lists; with
// DIAG of one list, j < k.
template <bool DIAG>
__device__ __forceinline__ void near_block(const NearPipe& N, int j0, int j1, int k, float kx, float ky, float kz,
                                           uint32_t Uq, uint32_t rs, uint32_t dump, const NearParams& p) {
    const f32x2 X = splat2(kx), Y = splat2(ky), Z = splat2(kz), scale = splat2(p.inv_bw), off = splat2(p.off);
    const uint32_t Um = Uq - (uint32_t)MAGIC_BITS * rs;
    for (int j = j0; j < j1; j += 4) {
        const float4 x4 = *reinterpret_cast<const float4*>(N.x + j), y4 = *reinterpret_cast<const float4*>(N.y + j),
                     z4 = *reinterpret_cast<const float4*>(N.z + j);
        const uint4 c4 = *reinterpret_cast<const uint4*>(N.code + j);
        const f32x2 xj[2] = {pk2(x4.x, x4.y), pk2(x4.z, x4.w)}, yj[2] = {pk2(y4.x, y4.y), pk2(y4.z, y4.w)},
                    zj[2] = {pk2(z4.x, z4.y), pk2(z4.z, z4.w)};
        const uint32_t cj[4] = {c4.x, c4.y, c4.z, c4.w};
        unsigned redo = 0;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const f32x2 dx = sub2(xj[h], X), dy = sub2(yj[h], Y), dz = sub2(zj[h], Z);
            const f32x2 d2 = fma2(dz, dz, fma2(dy, dy, mul2(dx, dx)));
            float s0, s1, e[2];
            uint32_t b[2];
            up2(d2, s0, s1);
            const f32x2 d = mul2(d2, pk2(rsqrt_approx(s0), rsqrt_approx(s1)));
            magic_bits2(fma2(d, scale, off), b[0], b[1], e[0], e[1]);
#pragma unroll
            for (int t = 0; t < 2; t++) {
                const bool safe = fabsf(e[t]) <= p.thr;
                // (below a lower edge above 0: code 0)
                const bool take = safe && b[t] < MAGIC_BITS + (uint32_t)p.n && (!DIAG || j + 2 * h + t < k);
                count_at(take ? max(b[t], (uint32_t)MAGIC_BITS) * rs + (Um + cj[2 * h + t]) : dump);
                if (!safe) redo |= 1u << (2 * h + t);
            }
        }
        while (redo) {
            const int q = __ffs(redo) - 1, jj = j + q;
            redo &= redo - 1u;
            if (jj >= j1 || kx == -NEAR_PAD || (DIAG && jj >= k)) continue;
            const int r = near_exact(make_float4(N.x[jj], N.y[jj], N.z[jj], 0.f), make_float4(kx, ky, kz, 0.f), p);
            if (r >= 0) count_at((uint32_t)r * rs + Uq + N.code[jj]);
        }
    }
}

// One CTA per SM of `pipes` 8-warp pipelines around one shared accumulator.  A
// pipeline takes an item (a few centres of one tile), and waits for the others
// at a CTA barrier when its item belongs to another job, when there is none
// left, or when the 32-bit counters have taken NEAR_STOP pairs; there the
// counters are added to the job's accumulator.  A pipeline that draws just below
// the line still counts its item, so the line and an item of every pipeline
// have to stay below 2^32 counts of one word.  A centre has at most
// NEAR_MAX_POINTS^2 / 2 pairs of one list, but NEAR_MAX_POINTS^2 of two.
constexpr unsigned long long NEAR_STOP = 1ull << 30;
constexpr unsigned long long near_item_pairs(int centres, bool two_lists) {
    return (unsigned long long)centres * NEAR_MAX_POINTS * NEAR_MAX_POINTS / (two_lists ? 1 : 2);
}
static_assert(NEAR_STOP + TS_GROUPS_MAX * near_item_pairs(NEAR_ITEM, false) < (1ull << 32), "counters, one list");
static_assert(NEAR_STOP + TS_GROUPS_MAX * near_item_pairs(NEAR_ITEM_ORDERED, true) < (1ull << 32), "counters, two lists");

__global__ void __launch_bounds__(TS_GROUPS_MAX * TS_GROUP_THREADS, 1)
three_near_kernel(const DevJob* __restrict__ jobs, const uint32_t* __restrict__ item_off, int njobs, unsigned int item0,
                  unsigned int nitems, int centres, unsigned int* counter, unsigned int* dense, unsigned long long* work,
                  NearParams p, int pipes) {
    extern __shared__ __align__(16) unsigned char smem[];
    NearPipe* const pipe = reinterpret_cast<NearPipe*>(smem);
    unsigned int* const U = reinterpret_cast<unsigned int*>(pipe + pipes);
    __shared__ unsigned long long s_since, s_pairs;
    const NearStride st = near_stride(p.n);
    __shared__ unsigned int s_dump;
    const uint32_t ubase = shared_addr(U), dump = shared_addr(&s_dump);
    const int gi = threadIdx.x / TS_GROUP_THREADS, gt = threadIdx.x % TS_GROUP_THREADS, warp = gt >> 5, lane = gt & 31;
    const TsPipe pp{gt, warp, lane, 1 + gi};
    NearPipe& N = pipe[gi];
    const int parts = (TILE + centres - 1) / centres;  // items of a tile
    for (int b = threadIdx.x; b < st.words; b += blockDim.x) U[b] = 0;
    if (threadIdx.x == 0) s_since = s_pairs = 0;
    auto draw = [&]() {  // by the pipeline's first warp; nothing more once the launch is refused
        if (warp != 0) return;
        unsigned int t = 0;
        if (lane == 0) {  // (both on their way together: an item after the refusal is left undone)
            const unsigned int refused = *(volatile unsigned int*)dense;
            t = atomicAdd(counter, 1u);
            if (refused) t = TASK_NONE;
        }
        t = __shfl_sync(0xffffffffu, t, 0);
        uint4 it = make_uint4(TASK_NONE, 0, 0, 0);
        if (t < nitems) {
            t += item0;
            const int slot = find_job(item_off, njobs, t);
            const unsigned int l = t - item_off[slot];
            it = make_uint4((unsigned)slot, l / parts, (l % parts) * centres, 0);
        }
        if (lane == 0) {
            N.item = it;
            N.stop = s_since >= NEAR_STOP;
        }
    };
    draw();
    int cur = -1;
    const unsigned lt = (1u << lane) - 1u;
    for (;;) {
        __syncthreads();  // every pipeline waits here with an item of another job, or none
        if (cur >= 0) {
            unsigned long long* g = jobs[cur].hist;
            const int m = p.n + 1, m3 = near_words3(p.n);
            for (int b = threadIdx.x; b < m3 + m + 1; b += blockDim.x) {
                const int at = b < m3 ? (b / (m * m)) * st.r + (b / m % m) * st.q + b % m : st.u2 + (b - m3);
                const unsigned int u = U[at];
                if (u) {
                    U[at] = 0;
                    atomicAdd(g + b, (unsigned long long)u);
                }
            }
        }
        uint32_t next = TASK_NONE;
        for (int g2 = 0; g2 < pipes; g2++) next = min(next, pipe[g2].item.x);  // (TASK_NONE is the largest)
        if (next == TASK_NONE) break;  // uniform: every thread read the same words
        __syncthreads();
        if (threadIdx.x == 0) s_since = 0;
        if (gt == 0) N.stop = 0;
        __syncthreads();
        cur = (int)next;
        const DevJob& J = jobs[cur];
        const uint32_t cls = J.mode & NEAR_CLASS_MASK;
        const int nlists = cls == NEAR_ORDERED ? 2 : 1;
        for (;;) {
            const uint4 item = N.item;
            if (item.x != next || N.stop) break;
            const int tile = (int)item.y, a0 = J.tile_start[0][tile], nA = J.tile_start[0][tile + 1] - a0;
            // tiles of each list within reach of the centre's tile
            if (gt < 2) N.ntiles[gt] = 0;
            pp.sync();
            const float4 *abox = J.box[0] + 2 * (size_t)tile;
            for (int l = 0; l < nlists; l++)
                for (int t = (cls == NEAR_SYM ? tile : 0) + gt; t < J.ntiles[1 + l]; t += TS_GROUP_THREADS)
                    if (boxes_near(abox, J.box[1 + l] + 2 * (size_t)t, p.reach2)) {
                        const int at = atomicAdd(&N.ntiles[l], 1);
                        if (at < NEAR_TILES) N.tiles[l][at] = (uint32_t)t;
                    }
            pp.sync();
            if (N.ntiles[0] > NEAR_TILES || N.ntiles[nlists - 1] > NEAR_TILES) {
                if (gt == 0) *dense = 1u;  // too many: the launch is counted by the tile kernel instead
            } else {
                // Entries of list l from its near tiles [t0, t1) at N[base ..),
                // at most cap of them; returns how many there are.  The codes
                // are scaled by `scale`; w: weight of the equal-index triples.
                auto build = [&](int l, int t0, int t1, int base, int cap, float4 c, int ci, unsigned w) -> int {
                    pp.sync();  // the pipeline is done with the list
                    if (gt == 0) N.count[l] = 0;
                    pp.sync();
                    for (int q = t0 + warp; q < t1; q += TS_WARPS) {
                        const int t = (int)N.tiles[l][q];
                        const float4 *bx = J.box[1 + l] + 2 * (size_t)t, lo = bx[0], hi = bx[1];
                        const float gx = fmaxf(0.f, fmaxf(lo.x - c.x, c.x - hi.x)), gy = fmaxf(0.f, fmaxf(lo.y - c.y, c.y - hi.y)),
                                    gz = fmaxf(0.f, fmaxf(lo.z - c.z, c.z - hi.z));
                        if ((gx * gx + gy * gy + gz * gz) * (1.0f - 4e-5f) >= p.reach2) continue;  // warp-uniform
                        const int b0 = J.tile_start[1 + l][t], nb = J.tile_start[1 + l][t + 1] - b0;
#pragma unroll
                        for (int r = 0; r < 2; r++) {
                            const int i = lane + 32 * r;
                            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                            int code = -1;
                            if (i < nb && !(cls == NEAR_SYM && t == tile && i <= ci)) {
                                v = J.pts[1 + l][b0 + i];
                                code = near_code(c, v, p);
                            }
                            const unsigned in = __ballot_sync(0xffffffffu, code >= 0);
                            if (!in) continue;
                            int at = 0;
                            if (lane == 0) at = atomicAdd(&N.count[l], __popc(in));
                            at = __shfl_sync(0xffffffffu, at, 0) + __popc(in & lt);
                            if (code >= 0) {
                                if (w) atomicAdd(U + st.u2 + code, w);
                                if (at < cap) {
                                    N.x[base + at] = v.x;
                                    N.y[base + at] = v.y;
                                    N.z[base + at] = v.z;
                                    N.code[base + at] = 4u * (uint32_t)code;
                                }
                            }
                        }
                    }
                    pp.sync();
                    const int n = N.count[l];
                    // padding to whole groups of four
                    if (gt < 4 && n + gt < cap && n + gt < ((n + 3) & ~3)) {
                        N.x[base + n + gt] = N.y[base + n + gt] = N.z[base + n + gt] = NEAR_PAD;
                        N.code[base + n + gt] = 0;
                    }
                    pp.sync();
                    return n;
                };
                // Every pair of entries j at [jb, jb + nj) and k at [kb, kb + nk);
                // tri: one list, j < k.  Blocks of 32 x 32 shared by the warps.
                auto pairs = [&](int jb, int nj, int kb, int nk, bool tri) {
                    const int bj = (nj + 31) / 32, bk = (nk + 31) / 32;
                    const int total = tri ? bk * (bk + 1) / 2 : bj * bk;
                    int kx = 0, jx = warp;  // block (jx, kx); tri: jx <= kx
                    for (int t = warp; t < total; t += TS_WARPS) {
                        while (jx >= (tri ? kx + 1 : bj)) {
                            jx -= tri ? kx + 1 : bj;
                            kx++;
                        }
                        const int k = kx * 32 + lane;
                        const bool in = k < nk;
                        const float x = in ? N.x[kb + k] : -NEAR_PAD, y = in ? N.y[kb + k] : -NEAR_PAD,
                                    z = in ? N.z[kb + k] : -NEAR_PAD;
                        const uint32_t Uq = ubase + (in ? N.code[kb + k] * (uint32_t)st.q : 0u);
                        const int j0 = jb + jx * 32, j1 = jb + min(nj, jx * 32 + 32);
                        if (tri && jx == kx) near_block<true>(N, j0, j1, kb + k, x, y, z, Uq, 4u * (uint32_t)st.r, dump, p);
                        else near_block<false>(N, j0, j1, 0, x, y, z, Uq, 4u * (uint32_t)st.r, dump, p);
                        jx += TS_WARPS;
                    }
                };
                unsigned long long done = 0;  // pairs of this item (all threads alike)
                for (int i = (int)item.z; i < min((int)item.z + centres, nA); i++) {
                    const float4 c = J.pts[0][a0 + i];
                    const unsigned w = cls == NEAR_SYM ? 2u : cls == NEAR_PAIR ? 1u : 0u;
                    if (cls == NEAR_SYM && gt == 0) atomicAdd(U + st.u2 + p.n + 1, 1u);
                    if (cls != NEAR_ORDERED) {
                        const int n = build(0, 0, N.ntiles[0], 0, NEAR_CAP, c, i, w);
                        done += (unsigned long long)n * (unsigned)max(n - 1, 0) / 2;
                        if (n <= NEAR_CAP) {
                            pairs(0, n, 0, n, true);
                        } else {
                            for (int u = 0; u < N.ntiles[0]; u += NEAR_CHUNK) {
                                const int nu = build(0, u, min(u + NEAR_CHUNK, N.ntiles[0]), 0, NEAR_CAP / 2, c, i, 0u);
                                pairs(0, nu, 0, nu, true);
                                for (int v = u + NEAR_CHUNK; v < N.ntiles[0]; v += NEAR_CHUNK) {
                                    const int nv = build(0, v, min(v + NEAR_CHUNK, N.ntiles[0]), NEAR_CAP / 2, NEAR_CAP / 2, c, i, 0u);
                                    pairs(0, nu, NEAR_CAP / 2, nv, false);
                                }
                            }
                        }
                    } else {
                        const int n0 = build(0, 0, N.ntiles[0], 0, NEAR_CAP / 2, c, i, 0u);
                        const int n1 = build(1, 0, N.ntiles[1], NEAR_CAP / 2, NEAR_CAP / 2, c, i, 0u);
                        done += (unsigned long long)n0 * (unsigned)n1;
                        if (n0 <= NEAR_CAP / 2 && n1 <= NEAR_CAP / 2) {
                            pairs(0, n0, NEAR_CAP / 2, n1, false);
                        } else {
                            for (int u = 0; u < N.ntiles[0]; u += NEAR_CHUNK) {
                                const int nu = build(0, u, min(u + NEAR_CHUNK, N.ntiles[0]), 0, NEAR_CAP / 2, c, i, 0u);
                                for (int v = 0; v < N.ntiles[1]; v += NEAR_CHUNK) {
                                    const int nv = build(1, v, min(v + NEAR_CHUNK, N.ntiles[1]), NEAR_CAP / 2, NEAR_CAP / 2, c, i, 0u);
                                    pairs(0, nu, NEAR_CAP / 2, nv, false);
                                }
                            }
                        }
                    }
                }
                if (gt == 0 && done) {
                    atomicAdd(&s_since, done);
                    atomicAdd(&s_pairs, done);
                }
            }
            pp.sync();  // the pipeline is done with the item and its list
            draw();
            pp.sync();
        }
    }
    if (threadIdx.x == 0 && s_pairs) atomicAdd(work, s_pairs);
}

// Sums over centres of products of their near counts, WB or WC, and the pair
// counts PBC: one warp per centre makes the two histograms, the CTA adds up the
// products.  hist: the sums (m x m, row: first list), aux: the pairs (m),
// weighted; with NEAR_SYM both lists are the same.
constexpr int WEDGE_ITEMS = TILE / TS_WARPS;  // items (TS_WARPS centres) of a tile

size_t three_wedge_smem_bytes(int n) { return (size_t)TS_WARPS * 2 * (n + 1) * sizeof(unsigned int); }

__global__ void __launch_bounds__(TS_GROUP_THREADS)
three_wedge_kernel(const DevJob* __restrict__ jobs, const uint32_t* __restrict__ item_off, int njobs,
                   unsigned int nitems, const unsigned int* __restrict__ dense, NearParams p) {
    const unsigned int refused = *dense;
    extern __shared__ __align__(16) unsigned char smem[];
    unsigned int* const H = reinterpret_cast<unsigned int*>(smem);  // [warp][list][code]
    __shared__ int s_job;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, m = p.n + 1;
    for (unsigned int t = blockIdx.x; t < nitems; t += gridDim.x) {
        __syncthreads();
        if (warp == 0) {
            const int slot = find_job(item_off, njobs, t);
            if (lane == 0) s_job = slot;
        }
        for (int b = threadIdx.x; b < TS_WARPS * 2 * m; b += blockDim.x) H[b] = 0;
        if (refused) return;  // (by the launch before this one: the same for all threads)
        __syncthreads();
        const DevJob& J = jobs[s_job];
        const unsigned int l = t - item_off[s_job];
        const int tile = (int)(l / WEDGE_ITEMS), a0 = J.tile_start[0][tile], nA = J.tile_start[0][tile + 1] - a0;
        const int i = (int)(l % WEDGE_ITEMS) * TS_WARPS + warp;
        const bool sym = (J.mode & NEAR_CLASS_MASK) == NEAR_SYM;
        if (i < nA) {
            const float4 c = J.pts[0][a0 + i];
            for (int x = 0; x < (sym ? 1 : 2); x++) {
                unsigned int* h = H + (warp * 2 + x) * m;
                for (int q0 = 0; q0 < J.ntiles[1 + x]; q0 += 32) {
                    bool near = false;
                    if (q0 + lane < J.ntiles[1 + x]) {
                        const float4 *bx = J.box[1 + x] + 2 * (size_t)(q0 + lane), lo = bx[0], hi = bx[1];
                        const float gx = fmaxf(0.f, fmaxf(lo.x - c.x, c.x - hi.x)), gy = fmaxf(0.f, fmaxf(lo.y - c.y, c.y - hi.y)),
                                    gz = fmaxf(0.f, fmaxf(lo.z - c.z, c.z - hi.z));
                        near = !((gx * gx + gy * gy + gz * gz) * (1.0f - 4e-5f) >= p.reach2);
                    }
                    for (unsigned mask = __ballot_sync(0xffffffffu, near); mask; mask &= mask - 1u) {
                        const int q = q0 + __ffs(mask) - 1, b0 = J.tile_start[1 + x][q], nb = J.tile_start[1 + x][q + 1] - b0;
#pragma unroll
                        for (int r = 0; r < 2; r++)
                            if (lane + 32 * r < nb) {
                                const int code = near_code(c, J.pts[1 + x][b0 + lane + 32 * r], p);
                                if (code >= 0) atomicAdd(h + code, 1u);
                            }
                    }
                }
            }
        }
        __syncthreads();
        const int y = sym ? 0 : m;
        for (int e = threadIdx.x; e < m * m + m; e += blockDim.x) {
            unsigned long long s = 0;
            if (e < m * m) {
                for (int w = 0; w < TS_WARPS; w++)
                    s += (unsigned long long)H[w * 2 * m + e / m] * H[w * 2 * m + y + e % m];
                if (s) atomicAdd(J.hist + e, s);
            } else if (J.aux) {
                for (int w = 0; w < TS_WARPS; w++) s += H[w * 2 * m + y + (e - m * m)];
                if (s) atomicAdd(J.aux + (e - m * m), s * J.weight);
            }
        }
    }
}

// Expands accumulators (job: its hist) into the histograms (its aux): the
// orderings of each multiset, and in the reference's mode the triples with
// sides at or above hist_max.
__global__ void __launch_bounds__(256) three_expand_kernel(const DevJob* __restrict__ accs, NearParams p) {
    const DevJob& A = accs[blockIdx.y];
    const uint32_t cls = A.mode & NEAR_CLASS_MASK, centre = A.mode >> NEAR_CENTRE_SHIFT;
    const int n = p.n, m = n + 1, m3 = m * m * m, z = p.zcode, F = n + 1;
    const unsigned long long *U = A.hist, *U2 = U + m3, *WB = U2 + m + 1, *WC = WB + m * m, *P = WC + m * m;
    auto at = [&](int pp, int q, int r) { return U[(r * m + q) * m + pp]; };
    auto put = [&](int v0, int v1, int v2, unsigned long long u) {
        const long long x = ((long long)v2 * n + v1) * n + v0;
        if (x < p.len) atomicAdd(A.aux + x, u);
    };
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < m3 + 2 * m * m + m; e += gridDim.x * blockDim.x) {
        if (e < m3) {
            const int a = e % m, b = e / m % m, c = e / (m * m);
            unsigned long long u;
            if (cls == NEAR_SYM) {
                u = at(a, b, c) + at(a, c, b) + at(b, a, c) + at(b, c, a) + at(c, a, b) + at(c, b, a);
                if (a == z && b == c) u += U2[b];
                if (b == z && a == c) u += U2[a];
                if (c == z && a == b) u += U2[a];
                if (a == z && b == z && c == z) u += U2[m];
            } else if (cls == NEAR_PAIR) {
                if (centre == 0) u = at(a, b, c) + at(b, a, c) + (c == z && a == b ? U2[a] : 0ull);
                else if (centre == 1) u = at(a, c, b) + at(c, a, b) + (b == z && a == c ? U2[a] : 0ull);
                else u = at(b, c, a) + at(c, b, a) + (a == z && b == c ? U2[b] : 0ull);
            } else {
                u = at(a, b, c);
            }
            if (!u) continue;
            put(a, b, c, u);
            if (!p.clean) {
                put(a, F, c, 0ull - u);
                put(F, b, c, 0ull - u);
                put(F, F, c, u);
            }
        } else if (!p.clean) {
            const int k = e - m3;
            if (k < m * m) {
                const unsigned long long w = WB[k];
                if (w) {
                    put(k / m, F, k % m, w);
                    put(F, F, k % m, 0ull - w);
                    if (cls == NEAR_SYM) {
                        put(F, k / m, k % m, w);
                        put(F, F, k % m, 0ull - w);
                    }
                }
            } else if (k < 2 * m * m) {
                const unsigned long long w = WC[k - m * m];
                if (w) {
                    put(F, (k - m * m) / m, (k - m * m) % m, w);
                    put(F, F, (k - m * m) % m, 0ull - w);
                }
            } else if (P[k - 2 * m * m]) {
                put(F, F, k - 2 * m * m, P[k - 2 * m * m]);
            }
        }
    }
}

cudaError_t launch_three_near(const DevJob* jobs, const uint32_t* item_off, int njobs, unsigned int item0,
                              unsigned int nitems, int centres, unsigned int* counter, unsigned int* dense,
                              unsigned long long* work, const NearParams& p, int grid, int pipes, cudaStream_t st) {
    if (pipes < 1 || pipes > TS_GROUPS_MAX || centres < 1 || centres > NEAR_ITEM) return cudaErrorInvalidValue;
    three_near_kernel<<<grid, pipes * TS_GROUP_THREADS, three_near_smem_bytes(p.n, pipes), st>>>(
        jobs, item_off, njobs, item0, nitems, centres, counter, dense, work, p, pipes);
    return cudaGetLastError();
}

cudaError_t launch_three_wedges(const DevJob* jobs, const uint32_t* item_off, int njobs, unsigned int nitems,
                                const unsigned int* dense, const NearParams& p, int grid, cudaStream_t st) {
    if (nitems == 0) return cudaSuccess;
    three_wedge_kernel<<<std::min<unsigned int>(nitems, grid), TS_GROUP_THREADS, three_wedge_smem_bytes(p.n), st>>>(
        jobs, item_off, njobs, nitems, dense, p);
    return cudaGetLastError();
}

cudaError_t launch_three_expand(const DevJob* accs, int naccs, const NearParams& p, cudaStream_t st) {
    const int m = p.n + 1, words = m * m * m + 2 * m * m + m;
    // (at most 65535 accumulators a launch)
    for (int a = 0; a < naccs; a += 65535) {
        const dim3 grid(std::min(32, (words + 255) / 256), std::min(65535, naccs - a));
        three_expand_kernel<<<grid, 256, 0, st>>>(accs + a, p);
    }
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Pair counts (src/2pcf_C_version.cc).

constexpr int PR_WARPS = 8;
constexpr int PR_THREADS = PR_WARPS * 32;
constexpr int PR_CHUNK_MAX = 32;  // tiles B of one item at most (one mask word)
constexpr size_t PR_SMEM_FIXED = 2 * TILE * sizeof(float4);

// Tile A of an item, by coordinate, so that four points of one coordinate come
// in one 16-byte load; points past the end are NaN.
struct PairTile {
    float x[TILE], y[TILE], z[TILE];
    int key[TILE];
};
static_assert(sizeof(PairTile) + 4 <= PR_SMEM_FIXED, "pair tile and dump word");

// The reference's pair bin of the separation a-b, -1 if not counted.
template <bool FP64>
__device__ __forceinline__ int pair_bin(float4 a, float4 b, const PairParams& p) {
    const int bn = ref_bin_tp<FP64>(ref_dist<FP64>(a, b), p.lo, p.hi, p.n, 0);
    return bn >= 0 && bn < p.n ? bn : -1;
}

// Which pairs of two tiles count: every one, positions j >= i of one tile
// (self pairs are counted, as the reference's j >= i), or loop indices j >= i.
enum PairKind : int { PK_ALL = 0, PK_DIAG = 1, PK_KEY = 2 };

// Counts points [i0, i1) of tile A (i0 a multiple of 4) against tile B, whose
// points lane and lane + 32 each lane holds.  Guarded FP32: the squared
// separations of two points i run in packed f32x2 instructions, the bin
// coordinate comes from rsqrt.approx, and a coordinate inside the guard band
// around a bin edge -- or NaN: zero separations, padded and NaN points -- goes
// to the reference's formula.  Issue-bound: about 14 lane-instructions a pair
// instead of 57 with exact square roots and threshold lookups for every pair.
template <bool FP64, int KIND>
__device__ __forceinline__ void pair_tiles(const PairTile& A, int i0, int i1, const float4 (&pj)[2], int nB,
                                           const PairParams& p, unsigned int* Hw) {
    const int lane = threadIdx.x & 31;
    auto counted = [&](int i, int r) -> bool {
        if (KIND == PK_DIAG) return lane + 32 * r >= i;
        if (KIND == PK_KEY) return pkey(pj[r]) >= A.key[i];
        return true;
    };
    auto exact = [&](int i, int r) {
        if (i >= i1 || lane + 32 * r >= nB || !counted(i, r)) return;
        const int b = pair_bin<FP64>(make_float4(A.x[i], A.y[i], A.z[i], 0.f), pj[r], p);
        if (b >= 0) atomicAdd(Hw + b, 1u);
    };
    if (FP64 || !p.fast) {
        for (int i = i0; i < i1; i++) {
            exact(i, 0);
            exact(i, 1);
        }
        return;
    }
    const f32x2 X[2] = {splat2(pj[0].x), splat2(pj[1].x)}, Y[2] = {splat2(pj[0].y), splat2(pj[1].y)},
                Z[2] = {splat2(pj[0].z), splat2(pj[1].z)};
    const f32x2 scale = splat2(p.inv_bw), off = splat2(p.off);
    const uint32_t base = shared_addr(Hw) - 4u * MAGIC_BITS, n = (uint32_t)p.n;
    const uint32_t dump = shared_addr(&A + 1);  // (the tile fills half of PR_SMEM_FIXED)
    for (int i = i0; i < i1; i += 4) {
        const float4 x4 = *reinterpret_cast<const float4*>(A.x + i), y4 = *reinterpret_cast<const float4*>(A.y + i),
                     z4 = *reinterpret_cast<const float4*>(A.z + i);
        const f32x2 xi[2] = {pk2(x4.x, x4.y), pk2(x4.z, x4.w)}, yi[2] = {pk2(y4.x, y4.y), pk2(y4.z, y4.w)},
                    zi[2] = {pk2(z4.x, z4.y), pk2(z4.z, z4.w)};
        unsigned redo = 0;  // bit 4 h + 2 t + r: pair (i + 2 h + t, lane + 32 r) near a bin edge
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const f32x2 dx = sub2(xi[h], X[r]), dy = sub2(yi[h], Y[r]), dz = sub2(zi[h], Z[r]);
                const f32x2 d2 = fma2(dz, dz, fma2(dy, dy, mul2(dx, dx)));
                float s0, s1, e[2];
                uint32_t b[2];
                up2(d2, s0, s1);
                const f32x2 d = mul2(d2, pk2(rsqrt_approx(s0), rsqrt_approx(s1)));
                magic_bits2(fma2(d, scale, off), b[0], b[1], e[0], e[1]);
#pragma unroll
                for (int t = 0; t < 2; t++) {
                    const bool safe = fabsf(e[t]) <= p.thr;
                    const bool take = safe && b[t] - MAGIC_BITS < n && counted(i + 2 * h + t, r);
                    count_at(take ? base + 4u * b[t] : dump);
                    if (!safe) redo |= 1u << (4 * h + 2 * t + r);
                }
            }
        while (redo) {
            const int q = __ffs(redo) - 1;
            redo &= redo - 1u;
            exact(i + (q >> 1), q & 1);
        }
    }
}

template <bool FP64>
__device__ __forceinline__ void pair_tiles_kind(int kind, const PairTile& A, int i0, int i1, const float4 (&pj)[2],
                                                int nB, const PairParams& p, unsigned int* Hw) {
    if (kind == PK_DIAG) pair_tiles<FP64, PK_DIAG>(A, i0, i1, pj, nB, p, Hw);
    else if (kind == PK_KEY) pair_tiles<FP64, PK_KEY>(A, i0, i1, pj, nB, p, Hw);
    else pair_tiles<FP64, PK_ALL>(A, i0, i1, pj, nB, p, Hw);
}

// Runs f(q, i0, i1) for this warp's share of n tiles B against nA points of
// tile A: with few tiles B the points of A are shared out too.
template <typename F>
__device__ __forceinline__ void pair_share(int n, int nA, F&& f) {
    const int warp = threadIdx.x >> 5;
    const int split = n >= 2 * PR_WARPS ? 1 : (n >= PR_WARPS ? 2 : (n >= 4 ? 4 : 8)), len = TILE / split;
    for (int u = warp; u < n * split; u += PR_WARPS) {
        const int i0 = (u % split) * len;
        if (i0 < nA) f(u / split, i0, min(i0 + len, nA));
    }
}

// Persistent over items (job, tile A, chunk of tiles B); the first warp draws
// the next item with tiles B in reach, stages its tile A and leaves the mask of
// those tiles; the warps share the tiles B out, each keeping its tile's points
// in registers.  No task list: an item is its index, its tiles are tested
// here against the views' boxes.
template <bool FP64>
__global__ void __launch_bounds__(PR_THREADS, PAIR_CTAS)
pair_kernel(const DevJob* __restrict__ jobs, const uint32_t* __restrict__ item_off, int njobs, unsigned int item0,
            unsigned int nitems, int chunk, unsigned int* counter, unsigned long long* work, PairParams p, int copies) {
    extern __shared__ __align__(16) unsigned char smem[];
    PairTile& A = *reinterpret_cast<PairTile*>(smem);
    unsigned int* H = reinterpret_cast<unsigned int*>(smem + PR_SMEM_FIXED);
    __shared__ int4 s_item;  // job (-1: none), first tile B, mask of tiles B, tile A
    for (int b = threadIdx.x; b < copies * p.n; b += blockDim.x) H[b] = 0;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned int* Hw = H + (warp % copies) * p.n;
    unsigned long long pairs = 0;   // lanes of the first warp
    unsigned int tile_pairs = 0;
    int cur = -1;
    unsigned int since = 0;
    for (;;) {
        __syncthreads();
        if (warp == 0) {
            int4 it = make_int4(-1, 0, 0, 0);
            for (;;) {
                unsigned int t = 0;
                if (lane == 0) t = atomicAdd(counter, 1u);
                t = __shfl_sync(0xffffffffu, t, 0);
                if (t >= nitems) break;
                t += item0;
                const int slot = find_job(item_off, njobs, t);
                const DevJob& J = jobs[slot];
                const unsigned int nbc = (unsigned int)(J.ntiles[1] + chunk - 1) / chunk, l = t - item_off[slot];
                const int a = (int)(l / nbc), b0 = (int)(l % nbc) * chunk, b = b0 + lane;
                const bool near = lane < chunk && b < J.ntiles[1] && (!(J.mode & JOB_B_FROM_A) || b >= a) &&
                                  boxes_near(J.box[0] + 2 * (size_t)a, J.box[1] + 2 * (size_t)b, p.reach2);
                const unsigned int mask = __ballot_sync(0xffffffffu, near);
                if (!mask) continue;
                const int a0 = J.tile_start[0][a], nA = J.tile_start[0][a + 1] - a0;
                if (near) {
                    const unsigned int nB = (unsigned int)(J.tile_start[1][b + 1] - J.tile_start[1][b]);
                    pairs += (J.mode & JOB_B_FROM_A) && b == a ? (unsigned)nA * ((unsigned)nA + 1u) / 2u : (unsigned)nA * nB;
                    tile_pairs++;
                }
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    const int i = lane + 32 * r;
                    const float4 v = i < nA ? J.pts[0][a0 + i] : make_float4(NAN, NAN, NAN, 0.f);
                    A.x[i] = v.x;
                    A.y[i] = v.y;
                    A.z[i] = v.z;
                    A.key[i] = pkey(v);
                }
                it = make_int4(slot, b0, (int)mask, a);
                break;
            }
            if (lane == 0) s_item = it;
        }
        __syncthreads();
        const int4 it = s_item;
        // (an item adds at most 32 x 64^2 counts to a bin: 4096 items keep the 32-bit counters below 2^30)
        if ((it.x != cur || since >= 4096) && cur >= 0) {
            flush_hist(H, copies, p.n, jobs[cur].hist);
            since = 0;
        }
        cur = it.x;
        if (cur < 0) break;
        since++;
        const DevJob& J = jobs[cur];
        const int nA = J.tile_start[0][it.w + 1] - J.tile_start[0][it.w];
        unsigned int left = (unsigned int)it.z;
        int at = 0;  // tiles of the mask taken from `left`
        pair_share(__popc((unsigned int)it.z), nA, [&](int q, int i0, int i1) {
            for (; at < q; at++) left &= left - 1u;
            const int b = it.y + __ffs(left) - 1;
            const int b0 = J.tile_start[1][b], nB = J.tile_start[1][b + 1] - b0;
            float4 pj[2];
#pragma unroll
            for (int r = 0; r < 2; r++)
                pj[r] = lane + 32 * r < nB ? J.pts[1][b0 + lane + 32 * r] : make_float4(NAN, NAN, NAN, 0.f);
            const int kind = (J.mode & JOB_PRED_MASK) == PRED_SAME ? PK_KEY
                             : (J.mode & JOB_B_FROM_A) && b == it.w ? PK_DIAG : PK_ALL;
            pair_tiles_kind<FP64>(kind, A, i0, i1, pj, nB, p, Hw);
        });
    }
    if (warp == 0) {
        if (pairs) atomicAdd(work, pairs);
        if (tile_pairs) atomicAdd(work + 1, (unsigned long long)tile_pairs);
    }
}

// ---------------------------------------------------------------------------
// Self-check of the exception table: counts floats whose table-driven value
// differs from the table entry (should be 0) -- used by tests.
__global__ void acos_check_kernel(AcosTable t, uint32_t key_begin, uint32_t count, unsigned int* mismatches) {
    for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < count; e += gridDim.x * blockDim.x) {
        uint32_t idx = key_begin + e;
        if (idx >= t.n) break;
        float c = __uint_as_float(t.keys[idx]);
        if (__float_as_uint(acosf_ref(c, t)) != t.vals[idx]) atomicAdd(mismatches, 1u);
    }
}

// ---------------------------------------------------------------------------
// Launchers

size_t triangle_smem_bytes(int hist_len, int copies, bool jbj) {
    return (tri_wide_queue(hist_len, jbj) ? TRI_SMEM_WIDE : TRI_SMEM_NARROW) + (size_t)hist_len * copies * 4;
}
size_t three_side_smem_bytes(const ThreeParams& p, int copies, int groups) {
    // groups > 0: the grouped kernel (one histogram); else 8-warp CTAs with
    // 'copies' copies (0: the global histogram)
    const size_t pipe = ts_layout(ts_byte_jk(p)).bytes;
    const int words = groups > 0 || copies > 0 ? hist_stride(ts_acc_words(p)) : 0;
    if (groups > 0) return (size_t)groups * pipe + (size_t)words * 4;
    return pipe + (size_t)words * copies * 4;
}
// Guard band of the fast pair bins.  With u = 2^-24 the reference's separation
// is within 2.5 u of the exact one of the same float differences and the fast
// one (packed FMAs, rsqrt.approx at 2^-22.9, one product) within 4.7 u; the
// subtraction of lo, the two divisions by bw and the fused coordinate add at
// most 5.5 u of the coordinate range D = max(|lo|, |hi|) / bw + 1: together
// below 12.7 u D = 7.6e-7 D bins.  The band is 1e-6 (D + 1).  Finer binnings
// than 2^16 steps go to the reference's formula pair by pair.
void pair_guard(PairParams& p) {
    const double D = std::max(fabs((double)p.lo), fabs((double)p.hi)) / (double)p.bw + 1.0;
    p.fast = D <= 65536.0 && p.bw >= 1e-30f ? 1 : 0;
    if (!p.fast) return;
    p.inv_bw = (float)(1.0 / (double)p.bw);
    p.off = (float)(-(double)p.lo / (double)p.bw - 0.5);
    p.thr = (float)(0.5 - 1e-6 * (D + 1.0));
}

// Tiles B per item of the pair kernels: as many as leave eight items to every
// resident CTA, at least one for each of its warps (an item's tile A is staged
// once, but the items are what balances the CTAs).  One where there are few tile
// pairs for the CTAs, whose warps then share the points of tile A (1,500 points,
// DD + DR: 21 us with eight, 17 with one), and in FP64, where a tile pair is 30 us
// (6,000 points 2.0 and 1.0 ms).
int pair_chunk(long long tile_pairs, int ctas, bool fp64) {
    if (fp64 || tile_pairs < 2ll * ctas) return 1;
    int chunk = PR_CHUNK_MAX;
    while (chunk > PR_WARPS && tile_pairs / chunk < 8ll * ctas) chunk /= 2;
    return chunk;
}

size_t pair_smem_bytes(int hist_len, int copies) { return PR_SMEM_FIXED + (size_t)hist_len * copies * 4; }

// Every counting kernel may use the device's whole opt-in shared memory per
// block.  Set once per device, before any launch or graph capture, and never
// lowered: a launch (or a captured graph replayed later) is then valid for
// any histogram size the launch shape allows.
cudaError_t prepare_kernels(int device) {
    int optin = 0;
    cudaError_t e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
    if (e != cudaSuccess) return e;
    const void* fns[] = {(const void*)triangle_fast_kernel<true, FAST_TP, uint32_t>,
                         (const void*)triangle_fast_kernel<false, FAST_TP, uint32_t>,
                         (const void*)triangle_fast_kernel<false, FAST_GEOM, uint32_t>,
                         (const void*)triangle_fast_kernel<false, FAST_TP, uint16_t>,
                         (const void*)triangle_fast_kernel<false, FAST_JBJ, uint16_t>,
                         (const void*)triangle_fast_kernel<false, FAST_GEOM, uint16_t>,
                         (const void*)triangle_fp64_kernel<MODE_FP64>, (const void*)triangle_fp64_kernel<MODE_GEOM>,
                         (const void*)triangle_fp64_kernel<MODE_JBJ>, (const void*)three_side_kernel<true, true>,
                         (const void*)three_side_kernel<true, false>, (const void*)three_side_kernel<false, true>,
                         (const void*)three_side_kernel<false, false>, (const void*)three_side_grouped_kernel<true>,
                         (const void*)three_side_grouped_kernel<false>, (const void*)pair_kernel<true>,
                         (const void*)pair_kernel<false>, (const void*)three_near_kernel, (const void*)three_wedge_kernel,
                         (const void*)tri_list_kernel<FAST_TP>, (const void*)tri_list_kernel<FAST_JBJ>,
                         (const void*)tri_list_kernel<FAST_GEOM>};
    for (const void* f : fns) {
        cudaFuncAttributes fa;
        e = cudaFuncGetAttributes(&fa, f);
        if (e != cudaSuccess) return e;
        // dynamic plus static shared memory may not exceed the opt-in limit
        e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)fa.sharedSizeBytes);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_triangle_fast(const DevJob* jobs, UnitList ul, unsigned int* counter, const TriParams& p,
                                 RecheckQueue q, int grid, int copies, int mode, cudaStream_t st) {
    const size_t smem = triangle_smem_bytes(p.len, copies, mode == FAST_JBJ);
    const bool wide = tri_wide_queue(p.len, false);
    auto kern = mode == FAST_JBJ    ? triangle_fast_kernel<false, FAST_JBJ, uint16_t>
                : mode == FAST_GEOM ? (wide ? triangle_fast_kernel<false, FAST_GEOM, uint32_t> : triangle_fast_kernel<false, FAST_GEOM, uint16_t>)
                : !wide             ? triangle_fast_kernel<false, FAST_TP, uint16_t>
                : p.theta_full      ? triangle_fast_kernel<true, FAST_TP, uint32_t>
                                    : triangle_fast_kernel<false, FAST_TP, uint32_t>;
    kern<<<grid, TRI_THREADS, smem, st>>>(jobs, ul, counter, p, q, copies);
    return cudaGetLastError();
}

cudaError_t launch_triangle_recheck(const DevJob* jobs, RecheckQueue q, const TriParams& p, AcosTable t, int mode,
                                    int grid, cudaStream_t st) {
    auto kern = mode == FAST_JBJ ? triangle_recheck_kernel<FAST_JBJ> : mode == FAST_GEOM ? triangle_recheck_kernel<FAST_GEOM>
                                                                                         : triangle_recheck_kernel<FAST_TP>;
    kern<<<grid, 128, 0, st>>>(jobs, q, p, t);
    return cudaGetLastError();
}

cudaError_t launch_triangle_fp64(const DevJob* jobs, UnitList ul, unsigned int* counter, const TriParams& p,
                                 AcosTable t, int grid, int copies, int mode, cudaStream_t st) {
    const size_t smem = triangle_smem_bytes(p.len, copies, mode == MODE_JBJ);
    auto kern = mode == MODE_GEOM ? triangle_fp64_kernel<MODE_GEOM>
                : mode == MODE_JBJ  ? triangle_fp64_kernel<MODE_JBJ>
                                    : triangle_fp64_kernel<MODE_FP64>;
    kern<<<grid, TRI_THREADS, smem, st>>>(jobs, ul, counter, p, t, copies);
    return cudaGetLastError();
}

cudaError_t launch_three_side(const DevJob* jobs, UnitList ul, unsigned int* counter, const ThreeParams& p, int fp64,
                              int grid, int copies, int groups, cudaStream_t st) {
    if (groups > 0) {
        if (groups > TS_GROUPS_MAX) return cudaErrorInvalidValue;
        const size_t smem = three_side_smem_bytes(p, 1, groups);
        const int threads = groups * TS_GROUP_THREADS;
        if (fp64)
            three_side_grouped_kernel<true><<<grid, threads, smem, st>>>(jobs, ul, counter, p, groups);
        else
            three_side_grouped_kernel<false><<<grid, threads, smem, st>>>(jobs, ul, counter, p, groups);
        return cudaGetLastError();
    }
    const bool global = copies == 0;
    const size_t smem = three_side_smem_bytes(p, global ? 0 : copies, 0);
#define TS_LAUNCH(FP, GL) \
    three_side_kernel<FP, GL><<<grid, TS_GROUP_THREADS, smem, st>>>(jobs, ul, counter, p, copies > 0 ? copies : 1);
    if (fp64) {
        if (global) { TS_LAUNCH(true, true) } else { TS_LAUNCH(true, false) }
    } else {
        if (global) { TS_LAUNCH(false, true) } else { TS_LAUNCH(false, false) }
    }
#undef TS_LAUNCH
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Catalog conversion (sample_data/gen_flat_MICE_data.py:53-99): comoving
// distance from redshift by the quadratic fit r = p0 + p1 z + p2 z^2, then
//   x = r sin(rad (90 - dec)) sin(rad ra), y = r sin(rad (90 - dec)) cos(rad ra),
//   z = r cos(rad (90 - dec)),  rad = pi/180,
// in double with the script's order of operations (no contraction), rounded
// to the float coordinates the counting kernels use.
__global__ void radecz_kernel(const double* __restrict__ ra, const double* __restrict__ dec,
                              const double* __restrict__ zr, int64_t n, double p0, double p1, double p2,
                              float* __restrict__ x, float* __restrict__ y, float* __restrict__ z) {
    const double rad = 3.141592653589793 / 180.0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double zz = zr[i];
        const double r = __dadd_rn(__dadd_rn(p0, __dmul_rn(p1, zz)), __dmul_rn(__dmul_rn(p2, zz), zz));
        const double polar = __dmul_rn(rad, __dsub_rn(90.0, dec[i]));
        const double az = __dmul_rn(rad, ra[i]);
        double sp, cp, sa, ca;
        sincos(polar, &sp, &cp);
        sincos(az, &sa, &ca);
        const double rs = __dmul_rn(r, sp);
        x[i] = __double2float_rn(__dmul_rn(rs, sa));
        y[i] = __double2float_rn(__dmul_rn(rs, ca));
        z[i] = __double2float_rn(__dmul_rn(r, cp));
    }
}

cudaError_t launch_radecz_to_xyz(const double* ra, const double* dec, const double* redshift, int64_t n,
                                 const double poly[3], float* x, float* y, float* z, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    int64_t blocks = std::min<int64_t>((n + 255) / 256, 152 * 16);
    radecz_kernel<<<(unsigned)blocks, 256, 0, st>>>(ra, dec, redshift, n, poly[0], poly[1], poly[2], x, y, z);
    return cudaGetLastError();
}

cudaError_t launch_pairs(const DevJob* jobs, const uint32_t* item_off, int njobs, unsigned int item0,
                         unsigned int nitems, int chunk, unsigned int* counter, unsigned long long* work,
                         const PairParams& p, int fp64, int grid, int copies, cudaStream_t st) {
    if (chunk < 1 || chunk > PR_CHUNK_MAX) return cudaErrorInvalidValue;
    size_t smem = pair_smem_bytes(p.n, copies);
    if (fp64)
        pair_kernel<true><<<grid, PR_THREADS, smem, st>>>(jobs, item_off, njobs, item0, nitems, chunk, counter, work, p,
                                                          copies);
    else
        pair_kernel<false><<<grid, PR_THREADS, smem, st>>>(jobs, item_off, njobs, item0, nitems, chunk, counter, work,
                                                           p, copies);
    return cudaGetLastError();
}

cudaError_t launch_acos_check(AcosTable t, uint32_t key_begin, uint32_t count, unsigned int* mismatches,
                              cudaStream_t st) {
    acos_check_kernel<<<1024, 256, 0, st>>>(t, key_begin, count, mismatches);
    return cudaGetLastError();
}

}  // namespace tpcf

// ===========================================================================
// Pair counts without any device allocation.
//
// For callers that cannot call cudaMalloc -- code running inside a framework
// that owns all device memory through its own pool, or a library that must not
// grow the process's footprint behind its host application's back.  They pass
// device pointers to their catalogs and to the output histogram; the kernel
// reads the coordinates where they are and needs no other buffer, so that
// calls may overlap.  At most NOALLOC_MAX_POINTS points per catalog.
// ===========================================================================

namespace tpcf {

constexpr int64_t NOALLOC_MAX_POINTS = 1 << 18;             // per catalog

// Pair counts straight from coordinate arrays: tiles are runs of 64 points,
// item t is tile A t / nbc with chunk t % nbc of tiles B (from tile A on with
// 'same': one catalog, j >= i), handed out in grid strides (without spatial
// order every tile pair costs the same), so that neither a packed copy, a
// task list nor a counter is needed.
__global__ void __launch_bounds__(PR_THREADS, PAIR_CTAS)
pair_kernel_noalloc(const float* __restrict__ x0, const float* __restrict__ y0, const float* __restrict__ z0, int n0,
                    const float* __restrict__ x1, const float* __restrict__ y1, const float* __restrict__ z1, int n1,
                    int same, int pred_same, int chunk, PairParams p, int copies, unsigned long long* hist) {
    extern __shared__ __align__(16) unsigned char smem[];
    PairTile& A = *reinterpret_cast<PairTile*>(smem);
    unsigned int* H = reinterpret_cast<unsigned int*>(smem + PR_SMEM_FIXED);
    for (int b = threadIdx.x; b < copies * p.n; b += blockDim.x) H[b] = 0;
    const int lane = threadIdx.x & 31;
    unsigned int* Hw = H + ((threadIdx.x >> 5) % copies) * p.n;
    const int ntA = (n0 + TILE - 1) / TILE, ntB = (n1 + TILE - 1) / TILE, nbc = (ntB + chunk - 1) / chunk;
    // (at most 2^18 points per catalog: a CTA's counters stay below 2^32 unless
    // one bin of a CTA collects a sixteenth of all 2^36 pairs: flush in between)
    unsigned int since = 0;
    for (int t = blockIdx.x; t < ntA * nbc; t += gridDim.x) {
        const int a = t / nbc, b0 = (same ? a : 0) + (t % nbc) * chunk, nb = min(chunk, ntB - b0);
        if (nb <= 0) continue;
        if (++since > 4096) {
            flush_hist(H, copies, p.n, hist);
            since = 1;
        }
        const int a0 = a * TILE, nA = min(TILE, n0 - a0);
        __syncthreads();  // the previous item is done with tile A
        if (threadIdx.x < TILE) {
            const int i = threadIdx.x;
            const bool in = i < nA;
            A.x[i] = in ? x0[a0 + i] : NAN;
            A.y[i] = in ? y0[a0 + i] : NAN;
            A.z[i] = in ? z0[a0 + i] : NAN;
            A.key[i] = a0 + i;
        }
        __syncthreads();
        pair_share(nb, nA, [&](int q, int i0, int i1) {
            const int b = b0 + q, j0 = b * TILE, nB = min(TILE, n1 - j0);
            float4 pj[2];
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const int j = lane + 32 * r;
                pj[r] = j < nB ? make_float4(x1[j0 + j], y1[j0 + j], z1[j0 + j], __int_as_float(j0 + j))
                               : make_float4(NAN, NAN, NAN, 0.f);
            }
            pair_tiles_kind<false>(pred_same ? PK_KEY : same && a == b ? PK_DIAG : PK_ALL, A, i0, i1, pj, nB, p, Hw);
        });
    }
    flush_hist(H, copies, p.n, hist);
}

}  // namespace tpcf

// Declared in include/tpcf.h.
extern "C" int32_t tpcf_pair_count_noalloc(const float* x0, const float* y0, const float* z0, int64_t n0,
                                           const float* x1, const float* y1, const float* z1, int64_t n1,
                                           int32_t loop, float lo, float hi, int32_t nbins, uint64_t* hist_out,
                                           void* stream) {
    using namespace tpcf;
    unsigned long long* hist = reinterpret_cast<unsigned long long*>(hist_out);
    if (n0 < 0 || n1 < 0 || n0 > NOALLOC_MAX_POINTS || n1 > NOALLOC_MAX_POINTS) return TPCF_ERR_INVALID;
    if (!hist || nbins <= 0 || !(hi > lo)) return TPCF_ERR_INVALID;
    if ((n0 > 0 && (!x0 || !y0 || !z0)) || (n1 > 0 && (!x1 || !y1 || !z1))) return TPCF_ERR_INVALID;
    if (loop != TPCF_LOOP_ALL && loop != TPCF_LOOP_SAME && loop != TPCF_LOOP_ONE) return TPCF_ERR_INVALID;
    int copies = 8;
    while (copies > 1 && pair_smem_bytes(nbins, copies) > 40 * 1024) copies /= 2;
    if (pair_smem_bytes(nbins, copies) > 227 * 1024) return TPCF_ERR_INVALID;
    // an error left by the caller's earlier work is reported, not consumed
    if (cudaPeekAtLastError() != cudaSuccess) return TPCF_ERR_CUDA;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return TPCF_ERR_NO_DEVICE;
    cudaStream_t st = (cudaStream_t)stream;
    // (an error of this call's own CUDA calls is consumed before returning, so
    // that it does not stay pending for the caller's next CUDA call)
    auto own_error = []() {
        (void)cudaGetLastError();
        return (int32_t)TPCF_ERR_CUDA;
    };
    if (cudaMemsetAsync(hist, 0, sizeof(unsigned long long) * (size_t)nbins, st) != cudaSuccess) return own_error();
    const bool same = loop == TPCF_LOOP_SAME && x0 == x1 && y0 == y1 && z0 == z1 && n0 == n1;
    const int pred_same = loop == TPCF_LOOP_SAME && !same;
    const int ntA = (int)((n0 + TILE - 1) / TILE), ntB = (int)((n1 + TILE - 1) / TILE);
    if (ntA > 0 && ntB > 0) {
        PairParams p;
        p.n = nbins;
        p.lo = lo;
        p.hi = hi;
        volatile float span = hi - lo;
        p.bw = span / (float)nbins;
        pair_guard(p);
        const size_t smem = pair_smem_bytes(nbins, copies);
        int sms = 0;
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return own_error();
        if (smem > 48 * 1024) {
            // the kernel's dynamic shared memory limit: always the device's opt-in
            // maximum, never lowered (a lower per-call value would invalidate
            // launches recorded earlier with a larger size); dynamic plus the
            // kernel's static shared memory within the opt-in limit
            int optin = 0;
            cudaFuncAttributes fa;
            if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
                cudaFuncGetAttributes(&fa, pair_kernel_noalloc) != cudaSuccess)
                return own_error();
            const int smem_max = optin - (int)fa.sharedSizeBytes;
            if ((size_t)smem_max < smem) return TPCF_ERR_INVALID;
            if (cudaFuncSetAttribute(pair_kernel_noalloc, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max) !=
                cudaSuccess)
                return own_error();
        }
        const int slots = sms * PAIR_CTAS, chunk = pair_chunk((long long)ntA * ntB, slots, false);
        const int nbc = (ntB + chunk - 1) / chunk;
        const int grid = (int)std::min<long long>((long long)ntA * nbc, slots);
        pair_kernel_noalloc<<<grid, PR_THREADS, smem, st>>>(x0, y0, z0, (int)n0, x1, y1, z1, (int)n1, same ? 1 : 0,
                                                            pred_same, chunk, p, copies, hist);
        if (cudaGetLastError() != cudaSuccess) return TPCF_ERR_CUDA;  // (consumed by the check itself)
    }
    return TPCF_OK;
}
