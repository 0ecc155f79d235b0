// engine.h -- internal structures shared by the host engine (engine.cpp) and
// the CUDA kernels (kernels.cu).  Not part of the public ABI (include/tpcf.h).
#ifndef TPCF_ENGINE_H
#define TPCF_ENGINE_H

#include <stdint.h>
#include <cuda_runtime.h>

namespace tpcf {

// Resident CTAs per SM of the pair kernels (their register budget).
constexpr int PAIR_CTAS = 5;

// Points per spatial tile.  A triangle task covers one tile of each role.
constexpr int TILE = 64;

// Per-triangle predicate of a task (how the reference's loop bounds restrict
// the triples of a tile triple).
enum Pred : uint32_t {
    PRED_NONE = 0,   // every triple of the tile triple counts once
    PRED_DDR = 1,    // weight [key_k >= key_i] + [key_k >= key_j]  (loop ONE, roles A == B)
    PRED_SAME = 2,   // key_i <= key_j <= key_k                      (loop SAME, generic arrays)
    PRED_ONE = 3,    // key_j <= key_k                               (loop ONE, generic arrays)
    PRED_RDD = 4     // weight [key_i >= key_j] + [key_i >= key_k]   (loop ONE, roles A == B, in the
                     // role order (C, A, A): the single-array point first; guarded kernel only)
};
// unit.x: bits 0..21 job slot, 22/23 quarter of the A tile's points, 24 whether
// the unit is that quarter only
constexpr uint32_t UNIT_SLOT_MASK = 0x3FFFFFu;
constexpr uint32_t MAX_BATCH_JOBS = UNIT_SLOT_MASK;  // jobs of one launch
constexpr int UNIT_QUARTER_SHIFT = 22;
constexpr uint32_t UNIT_QUARTER = 1u << 24;
// recheck queue item .x: job slot | weight << 22
constexpr int RECHECK_WEIGHT_SHIFT = 22;

// Per-side word of the fast triangle kernel: word = code16 * 128 + class_weight,
// in 16 bits, so that its j-k table holds it in two bytes.  code16 is the side's
// s-bin (monotone in the side length, so that those of the shortest and middle
// side are the min and median of the three words, >> 7; the kernel multiplies by
// Q*T); the special codes below keep that order.  The kernel takes binnings of at
// most MAX_FAST_S s bins (b == S, rounding at the top edge, stays below
// CODE16_ABOVE).  class_weight counts side classes so that the sum of a
// triangle's three weights tells whether any permutation can be counted: below
// s_lo: 4, at/above s_hi (or rounding to bin S): 1, in range: 0, zero length or
// at/above the largest side a counted triangle can have: 32 (rejects the triangle).
constexpr int CODE16_ZERO = -2, CODE16_BELOW = -1, CODE16_ABOVE = 255;
constexpr int CW_IN = 0, CW_ABOVE = 1, CW_BELOW = 4, CW_REJECT = 32;
constexpr int MAX_FAST_S = 254;
constexpr int MAX_TRI_BINS = (1 << 22) - 1;  // S*Q*T limit of the triangle kernels
// most A tiles in one window of the planner (one mask word)
constexpr int MAX_WINDOW = 32;
// weight sum (4*nBelow + nAbove, >= 32 if rejected) -> permutation validity
constexpr unsigned VALID_02 = 0x07u;    // shortest side in range (permutations 0 and 2)
constexpr unsigned VALID_1 = 0x33u;     // middle side in range, no zero side (permutation 1)

// A histogram target of one launch.
struct DevJob {
    const float4* pts[3];        // spatially sorted points of roles A, B, C; .w = loop index (int bits)
    const int32_t* tile_start[3];// tile -> first point, ntiles+1 entries
    const float4* box[3];        // tile bounding boxes: lo at 2 t, hi at 2 t + 1 (.w unused)
    int32_t ntiles[3];
    uint32_t mode;               // JOB_* bits
    unsigned long long* hist;    // global uint64 histogram (hist_len entries)
    unsigned long long* aux;     // three-side lists: see three_wedge_kernel, three_expand_kernel
    unsigned long long weight;
};
// the job's tile tuples and the predicate of its points
constexpr uint32_t JOB_PRED_MASK = 0x7u;   // Pred
constexpr uint32_t JOB_B_FROM_A = 8u;      // tiles B >= A of one view, positions j >= i (triangles: j > i) in a diagonal pair
constexpr uint32_t JOB_C_FROM_B = 16u;     // the same of tiles C and B, positions k and j

// Launch-wide binning constants for the triangle kernels.
struct TriParams {
    int S, Q, T, len;            // len = S*Q*T
    float s_lo, s_hi, s_bw;      // reference float values
    float q_lo, q_hi, q_bw;
    float t_lo, t_hi, t_bw;
    int nan_zero;
    // guarded fast path (all in units of bins)
    float q_scale;               // 1/q_bw
    float q_off;                 // -q_lo/q_bw - 0.5
    float q_thr;                 // 0.5 - guard half-width for q
    float t_coef[6];             // acos(|c|) ~ sqrt(1-|c|) * poly(|c|), scaled by 1/(pi' t_bw)
    float t_half;                // pi/(2 pi' t_bw)
    float t_off0;                // t_half - t_lo/t_bw - 0.5
    float t_thrA;                // 0.5 - fixed guard half-width for theta
    float t_thrB;                // slope of the c-dependent guard half-width
    float t2_off;                // (1 - 3 t_lo)/t_bw - 0.5 - 2*(-0.5) handled in code
    int theta_full;              // theta range covers (0,1): skip range checks
    float lmax;                  // sides >= lmax cannot belong to a counted triangle
    float mid_hi;                // s_hi * q_hi (rounded up; JBJ: s_hi / q_lo): a counted triangle has a side in the s
                                 // range and another below it (permutation 0/2: the middle one; 1: the longest)
    int tame;                    // every coordinate of the launch is a number of ordinary size
    float s_split, mid_split;    // a side within the s range and the limit of the next longer one (rounded up)
    // neighbour lists: squared reach of a centre, limit max(q S, top) of the
    // middle side given the shortest
    float list_r2, list_q, list_top;
    float list_t, list_q_thr;    // guard slope of an angle (JBJ: of theta), guard of a ratio
    // double-precision geometry: sides that are surely below s_lo / at or above
    // s_hi, the s coordinate (minus 0.5) and its guard, slope of the angle's
    float geo_s_below, geo_s_above, geo_s_inv, geo_s_off, geo_s_thr, geo_t;
};

constexpr int TS_UMAX = 68;  // squared-length thresholds of up to 64 bins

struct ThreeParams {
    int n;                       // nbins
    float lo, hi, bw;
    int clean;
    int len;                     // n^3
    // Side codes from squared lengths (guarded FP32 kernel, when fast != 0):
    // u[v] is the smallest float d2 whose reference bin sqrt(d2) -> v' has
    // v' >= v (v' = nbins + 1 for d >= hi), u[0] = -inf, u[nbins + 2] = NaN;
    // inv_bw ~ 1/bw gives a first guess within one bin of the answer.
    int fast;
    float inv_bw;
    float u[TS_UMAX];
    int zcode;  // bin of a zero-length side (nbins + 1 at or above hist_max)
};

struct PairParams {
    int n;
    float lo, hi, bw;
    // Guarded FP32 bins (when fast != 0): the coordinate d * inv_bw + off (bin
    // coordinate - 0.5) from an approximate square root is within 0.5 - thr
    // of the reference's; only values closer than that to a bin edge are
    // recomputed with the reference's formula.
    int fast = 0;
    float inv_bw = 0.f, off = 0.f, thr = 0.f;
    float reach2 = 0.f;  // tiles at least sqrt(reach2) apart hold no counted pair (rounded up)
};

// Three-side histogram from neighbour lists: the guard band of pair bins
// (PairParams), codes 0 .. n below hist_max.
struct NearParams {
    int n, len, clean, zcode;    // as ThreeParams
    float lo, hi, bw, inv_bw, off, thr;
    float reach2;                // squared: sides at or above it are at or above hist_max
};
// DevJob::mode of its jobs (roles: centre, first list, second list): which
// pairs of the lists make a triple, and the reference's role of the centre.
enum NearClass : uint32_t {
    NEAR_SYM = 0,      // one catalog: positions centre < j < k, every ordering
    NEAR_PAIR = 1,     // both lists of one catalog: unordered pairs, both orderings
    NEAR_ORDERED = 2   // every pair
};
constexpr uint32_t NEAR_CLASS_MASK = 3u;
constexpr int NEAR_CENTRE_SHIFT = 2;
// centres per item at most, where a batch has no NEAR_ORDERED job and where it
// has one (see NEAR_STOP: what the 32-bit counters hold)
constexpr int NEAR_ITEM = 4, NEAR_ITEM_ORDERED = 2;

// Exact glibc-acosf exception table on the device.
struct AcosTable {
    const uint32_t* keys;        // sorted float bit patterns of c
    const uint32_t* vals;        // glibc acosf(c) bit patterns
    const uint32_t* bucket;      // 65537 offsets by key >> 16
    uint32_t n;
};

// Guard-band recheck queue (device scratch).
struct RecheckQueue {
    uint4* items;                // {slot | weight << RECHECK_WEIGHT_SHIFT, ia, ib, ic}
    unsigned int* count;
    unsigned int cap;
    unsigned long long* hists;      // neighbour lists: the launch's first histogram
    unsigned long long* evaluated;  // triangles of (i,j) pairs the fast kernel walked
};

// Planner: which tile triples of a launch can hold a counted triple.
struct PlanParams {
    int window;        // A tiles per row (at most MAX_WINDOW)
    int per_tile;      // 1: a unit per A tile; 0: a unit per row and tile C, its A tiles as a mask
    int tri;           // test the s and q ranges on the triple's side bounds
    int max_parts;     // parts a heavy unit may be cut into: 1, 4 or (per_tile == 0) 16
    int slots;         // CTAs (pipelines) that will share the units
    float lmax2;       // squared: no counted triple has a side at or above it (infinite: no pruning)
    float s_lo2, s_hi2, q_hi2;
    float r, heavy;    // typical longest side of a counted triple; estimated triples above which a unit is heavy
};
// The plan of a launch, found on the device and kept while its batch repeats.
struct PlanHeader {
    uint32_t nunits;   // units to count (0 where they overflow the unit list)
    uint32_t needed;   // units found
    uint32_t parts;    // units each heavy one was cut into
    uint32_t mismatch; // not 0: the passes of the planner differed (the units are not valid)
    unsigned long long evaluated, tiles;  // triples and tile triples of the units
};
// row_off[j] .. row_off[j + 1]: rows (window of A tiles, tile B) of job j;
// row_cnt: two words per row; block_sum: plan_blocks(nrows) + 1 pairs of words
int plan_blocks(uint64_t nrows, int* rows_per_block);
cudaError_t launch_plan(const DevJob* jobs, const uint32_t* row_off, int njobs, uint32_t nrows, const PlanParams& pp,
                        uint2* row_cnt, uint2* block_sum, PlanHeader* header, uint4* units, uint32_t* masks,
                        uint32_t capacity, cudaStream_t st);

// ---- kernel launchers (kernels.cu) ----
cudaError_t prepare_kernels(int device);  // once per device before any launch
// The counting kernels take units [u0, u0 + n) of a plan; the fast triangle
// kernel's mode: 0 reference, 1 JBJ, 2 double-precision geometry
struct UnitList {
    const PlanHeader* header;
    const uint4* units;
    const uint32_t* masks;
    uint32_t u0, n;
};
cudaError_t launch_triangle_fast(const DevJob* jobs, UnitList ul, unsigned int* counter, const TriParams& p,
                                 RecheckQueue q, int grid, int hist_copies, int mode, cudaStream_t st);
cudaError_t launch_triangle_recheck(const DevJob* jobs, RecheckQueue q, const TriParams& p, AcosTable t,
                                    int mode, int grid, cudaStream_t st);
cudaError_t launch_triangle_fp64(const DevJob* jobs, UnitList ul, unsigned int* counter, const TriParams& p,
                                 AcosTable t, int grid, int hist_copies, int mode,
                                 cudaStream_t st);  // mode: 0 FP64, 1 geometry, 2 JBJ
cudaError_t launch_three_side(const DevJob* jobs, UnitList ul, unsigned int* counter, const ThreeParams& p, int fp64,
                              int grid, int hist_copies, int groups, cudaStream_t st);
// item_off[j] .. item_off[j + 1]: the items (tile A, chunk of `chunk` tiles B)
// of job j; counts items [item0, item0 + nitems); work[0], work[1] receive the
// pairs and tile pairs evaluated
cudaError_t launch_pairs(const DevJob* jobs, const uint32_t* item_off, int njobs, unsigned int item0,
                         unsigned int nitems, int chunk, unsigned int* counter, unsigned long long* work,
                         const PairParams& p, int fp64, int grid, int hist_copies, cudaStream_t st);
cudaError_t launch_acos_check(AcosTable t, uint32_t key_begin, uint32_t count, unsigned int* mismatches,
                              cudaStream_t st);
cudaError_t launch_radecz_to_xyz(const double* ra, const double* dec, const double* redshift, int64_t n,
                                 const double poly[3], float* x, float* y, float* z, cudaStream_t st);

// Triangle parametrizations from neighbour lists.  Its jobs (roles: centre,
// first list, second list; weight: the centre view's points and, from bit 32,
// the output slot) have in
// DevJob::mode the reference's predicate, whether both lists are one view's
// unordered pairs, and for centre and lists two bits each of the reference's
// role and of the rank that orders points of different views.
constexpr int TL_MAX_WARPS = 24;  // warps per SM of its register budget
constexpr uint32_t TL_SELF = 8u;
constexpr int TL_ROLE_SHIFT = 4, TL_RANK_SHIFT = 10;
cudaError_t launch_tri_list(const DevJob* jobs, const uint32_t* item_off, int njobs, unsigned int item0,
                            unsigned int nitems, int centres, int parts, int kparts, int hists, unsigned int* counter,
                            const TriParams& p, RecheckQueue q, int grid, int warps, int mode, cudaStream_t st);
size_t tri_list_smem_bytes(int hist_len, int hists, int warps);

// The three launches of a three-side neighbour-list count; *dense is set where the near
// tiles of a centre are too many (count with launch_three_side instead): no more
// is counted then.
cudaError_t launch_three_near(const DevJob* jobs, const uint32_t* item_off, int njobs, unsigned int item0,
                              unsigned int nitems, int centres, unsigned int* counter, unsigned int* dense,
                              unsigned long long* work, const NearParams& p, int grid, int pipes, cudaStream_t st);
cudaError_t launch_three_wedges(const DevJob* jobs, const uint32_t* item_off, int njobs, unsigned int nitems,
                                const unsigned int* dense, const NearParams& p, int grid, cudaStream_t st);
cudaError_t launch_three_expand(const DevJob* accs, int naccs, const NearParams& p, cudaStream_t st);
size_t three_near_acc_words(int n);
size_t three_near_smem_bytes(int n, int pipes);

// shared-memory bytes of a launch (for occupancy / admission)
size_t triangle_smem_bytes(int hist_len, int hist_copies, bool jbj);
size_t three_side_smem_bytes(const ThreeParams& p, int hist_copies, int groups);
size_t pair_smem_bytes(int hist_len, int hist_copies);
void pair_guard(PairParams& p);  // from p.n, lo, hi, bw
int pair_chunk(long long tile_pairs, int ctas, bool fp64);

}  // namespace tpcf
#endif
