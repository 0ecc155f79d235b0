// engine.cpp -- host side of the counting engine: the C ABI of include/tpcf.h.
//
// Responsibilities
//   * catalogs: host copy + device-resident float4 points;
//   * spatial views: a catalog range is reordered by a balanced k-d split into
//     tiles of exactly TILE points (last tile partial), each with an
//     axis-aligned bounding box; cached per (catalog, range);
//   * planning: the reference's loop nest becomes jobs of three views whose
//     tile triples (pairs, centres) the device finds.  Symmetric loop nests
//     (DDD/RRR: i<=j<=k over one array; DRR: j<=k over one array; DDR: i,j over
//     one array) are enumerated canonically so that each unordered set of
//     points is visited once; everything else as ordered tile triples with the
//     reference's index predicate evaluated per triangle.  Whether triangles
//     are counted from tiles or from neighbour lists is chosen per batch;
//   * launches: one persistent kernel per (kind, binning, precision) group,
//     then the exact recheck of guard-band triangles, then D2H of the counts;
//   * glibc acosf exception table for exact theta (built from the host libm by
//     an exhaustive scan of [-1, 1], cached on disk);
//   * serving: submit/wait with a worker thread that batches every pending job
//     of compatible binning into the next launch (continuous batching), with
//     admission by device-memory footprint.
#include "../../include/tpcf.h"
#include "engine.h"
#include "exact_acos.h"

#include <cuda_runtime.h>
#include <dlfcn.h>
#include <gnu/libc-version.h>
#include <math.h>
#include <stdio.h>
#include <string.h>
#include <sys/stat.h>
#include <unistd.h>

#include <algorithm>
#include <array>
#include <atomic>
#include <chrono>
#include <climits>
#include <cstdint>
#include <cmath>
#include <condition_variable>
#include <deque>
#include <functional>
#include <future>
#include <map>
#include <memory>
#include <mutex>
#include <numeric>
#include <string>
#include <thread>
#include <tuple>
#include <unordered_map>
#include <unordered_set>
#include <vector>

using namespace tpcf;

namespace {

thread_local std::string g_tls_error;
std::atomic<uint64_t> g_allocations{0};  // device and page-locked blocks taken from the driver so far

struct CudaError {
    cudaError_t e;
};

#define CK(x)                                             \
    do {                                                  \
        cudaError_t _e = (x);                             \
        if (_e != cudaSuccess) throw CudaError{_e};       \
    } while (0)

struct InvalidArg {
    std::string msg;
};
struct InternalError {
    std::string msg;
};

// ---------------------------------------------------------------------------
// device buffers

// Freed device blocks up to 64 MiB are kept per device and power-of-two size
// class for reuse (at most 2 GiB in all), so that the catalogs, views and
// task lists of a repeated upload-count-release cycle cost no cudaMalloc /
// cudaFree (each of which also synchronises the device).  A block is only
// freed once nothing can still use it: views and scratch buffers are released
// after the work that read them has completed on its stream.
class DeviceBlocks {
  public:
    static DeviceBlocks& get() {
        static DeviceBlocks* d = new DeviceBlocks();  // never destroyed: blocks live until the process ends
        return *d;
    }
    void* alloc(size_t bytes, size_t* cap) {
        if (bytes > limit_.load()) throw CudaError{cudaErrorMemoryAllocation};
        int dev = 0;
        CK(cudaGetDevice(&dev));
        size_t cls = 256;
        while (cls < bytes) cls <<= 1;
        if (cls > kMaxCached) {
            void* p = nullptr;
            g_allocations++;
            CK(cudaMalloc(&p, bytes));
            *cap = bytes;
            return p;
        }
        {
            std::lock_guard<std::mutex> lk(mu_);
            auto& v = free_[std::make_pair(dev, cls)];
            if (!v.empty()) {
                void* p = v.back();
                v.pop_back();
                cached_ -= cls;
                *cap = cls;
                return p;
            }
        }
        void* p = nullptr;
        g_allocations++;
        if (cudaMalloc(&p, cls) != cudaSuccess) {
            // out of memory: give the kept blocks back and try once more
            (void)cudaGetLastError();
            trim();
            CK(cudaMalloc(&p, cls));
        }
        *cap = cls;
        return p;
    }
    void trim() {
        std::lock_guard<std::mutex> lk(mu_);
        int dev = 0;
        cudaGetDevice(&dev);
        for (auto& kv : free_) {
            if (kv.first.first != dev) continue;
            for (void* q : kv.second) cudaFree(q);
            cached_ -= kv.first.second * kv.second.size();
            kv.second.clear();
        }
    }
    // larger blocks are refused as if memory had run out (tests)
    void set_limit(size_t bytes) { limit_.store(bytes); }
    void release(void* p, size_t cap) {
        if (!p) return;
        int dev = 0;
        if (cap <= kMaxCached && cudaGetDevice(&dev) == cudaSuccess) {
            std::lock_guard<std::mutex> lk(mu_);
            if (cached_ + cap <= kMaxTotal) {
                free_[std::make_pair(dev, cap)].push_back(p);
                cached_ += cap;
                return;
            }
        }
        cudaFree(p);
    }

  private:
    static constexpr size_t kMaxCached = (size_t)64 << 20, kMaxTotal = (size_t)2 << 30;
    std::mutex mu_;
    std::atomic<size_t> limit_{SIZE_MAX};
    std::map<std::pair<int, size_t>, std::vector<void*>> free_;
    size_t cached_ = 0;
};

template <typename T>
struct DevBuf {
    T* p = nullptr;
    size_t n = 0;
    size_t cap = 0;  // bytes of the block
    DevBuf() = default;
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
    ~DevBuf() { release(); }
    void release() {
        DeviceBlocks::get().release(p, cap);
        p = nullptr;
        n = 0;
        cap = 0;
    }
    void reserve(size_t m) {
        if (m <= n) return;
        release();
        p = (T*)DeviceBlocks::get().alloc(std::max<size_t>(m, 1) * sizeof(T), &cap);
        n = m;
    }
    size_t bytes() const { return n * sizeof(T); }
    void swap(DevBuf& o) {
        std::swap(p, o.p);
        std::swap(n, o.n);
        std::swap(cap, o.cap);
    }
};

// Page-locked host buffer (device-to-host copies inside captured graphs need one).
template <typename T>
struct PinnedBuf {
    T* p = nullptr;
    size_t n = 0;
    PinnedBuf() = default;
    PinnedBuf(const PinnedBuf&) = delete;
    PinnedBuf& operator=(const PinnedBuf&) = delete;
    ~PinnedBuf() { release(); }
    void release() {
        if (p) cudaFreeHost(p);
        p = nullptr;
        n = 0;
    }
    // grows to a power of two: cudaFreeHost waits for all work on the device,
    // so a serving lane that reallocated for every new batch size would wait
    // for the other lanes' kernels
    void reserve(size_t m) {
        if (m <= n) return;
        release();
        size_t c = 4096;
        while (c < m) c <<= 1;
        g_allocations++;
        CK(cudaMallocHost((void**)&p, c * sizeof(T)));
        n = c;
    }
};

struct Box {
    float lo[3], hi[3];
};

struct Catalog {
    std::vector<float> x, y, z;
    int64_t n = 0;
    bool tame = true;  // every coordinate a number of magnitude at most 1e15
};

struct View {
    uint64_t id = 0;  // unique per view object (plan cache key)
    int64_t n = 0;
    int ntiles = 0;
    DevBuf<float4> pts;          // sorted points, .w = loop index (int bits)
    DevBuf<int32_t> tile_start;  // ntiles + 1
    DevBuf<float4> box;          // tile boxes: lo at 2 t, hi at 2 t + 1
    std::vector<int32_t> h_tile_start;
    std::vector<Box> boxes;
    double extent = 0;        // mean widest side of its tiles' boxes
    size_t upload_bytes = 0;  // host-to-device bytes of its construction
    size_t bytes() const { return pts.bytes() + tile_start.bytes() + box.bytes(); }
};

// One split of order[lo, hi): along the widest axis, so that the left part
// holds a multiple of `tile` points.  Returns the split point, or -1 for a
// part of at most `tile` points (a leaf).
int64_t kd_split(const float* xyz, std::vector<int32_t>& order, int64_t lo, int64_t hi, int tile) {
    int64_t n = hi - lo;
    if (n <= tile) return -1;
    float mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (int64_t i = lo; i < hi; i++)
        for (int a = 0; a < 3; a++) {
            float v = xyz[3 * (int64_t)order[i] + a];
            mn[a] = std::min(mn[a], v);
            mx[a] = std::max(mx[a], v);
        }
    int ax = 0;
    for (int a = 1; a < 3; a++)
        if (mx[a] - mn[a] > mx[ax] - mn[ax]) ax = a;
    int64_t ntile = (n + tile - 1) / tile;
    int64_t left = ((ntile + 1) / 2) * tile;
    if (left >= n) left = n - tile;
    // the split coordinate beside each index, contiguous, so that the
    // selection compares without gathering from xyz (a NaN coordinate sorts
    // as +inf: the order stays a strict weak one)
    static thread_local std::vector<std::pair<float, int32_t>> keys;
    keys.resize((size_t)n);
    for (int64_t i = 0; i < n; i++) {
        const float v = xyz[3 * (int64_t)order[lo + i] + ax];
        keys[i] = {std::isnan(v) ? INFINITY : v, order[lo + i]};
    }
    std::nth_element(keys.begin(), keys.begin() + left, keys.begin() + n);  // (coordinate, index) order
    for (int64_t i = 0; i < n; i++) order[lo + i] = keys[i].second;
    return lo + left;
}

void parallel_items(size_t n, const std::function<void(size_t)>& fn);

// Balanced k-d split of order[0, n) until parts hold at most `tile` points;
// leaves appear in order, giving spatially compact tiles.  Level by level,
// the parts of a level split in parallel (each split is deterministic, so the
// order does not depend on the threads).
void kd_order(const float* xyz, std::vector<int32_t>& order, int64_t n, int tile) {
    std::vector<std::pair<int64_t, int64_t>> level{{0, n}};
    while (!level.empty()) {
        std::vector<int64_t> mids(level.size(), -1);
        auto split = [&](size_t i) { mids[i] = kd_split(xyz, order, level[i].first, level[i].second, tile); };
        if (level.size() < 4 || n < 4096) {
            for (size_t i = 0; i < level.size(); i++) split(i);
        } else {
            parallel_items(level.size(), split);
        }
        std::vector<std::pair<int64_t, int64_t>> next;
        for (size_t i = 0; i < level.size(); i++)
            if (mids[i] >= 0) {
                next.push_back({level[i].first, mids[i]});
                next.push_back({mids[i], level[i].second});
            }
        level.swap(next);
    }
}

// ---------------------------------------------------------------------------
// exact glibc acosf exception table

struct AcosHost {
    std::vector<uint32_t> keys, vals, bucket;
};

std::string cache_dir() {
    const char* env = getenv("TPCF_CACHE_DIR");
    if (env && *env) return env;
    Dl_info info;
    if (dladdr((void*)&cache_dir, &info) && info.dli_fname) {
        std::string p = info.dli_fname;
        size_t s = p.rfind('/');
        std::string dir = s == std::string::npos ? "." : p.substr(0, s);
        return dir + "/../_cache";
    }
    return "/tmp/tpcf_cache";
}

void mkdirs(const std::string& d) {
    std::string cur;
    for (size_t i = 0; i < d.size(); i++) {
        cur += d[i];
        if (d[i] == '/' && cur.size() > 1) mkdir(cur.c_str(), 0755);
    }
    mkdir(d.c_str(), 0755);
}

uint32_t fbits(float f) {
    uint32_t u;
    memcpy(&u, &f, 4);
    return u;
}
float ffrom(uint32_t u) {
    float f;
    memcpy(&f, &u, 4);
    return f;
}

// Exhaustive scan of every float c in [-1, 1]: record where the host libm's
// acosf differs from (float)tpcf_acos_d(c).
AcosHost build_acos_table() {
    const uint32_t spans[2][2] = {{0x00000000u, 0x3f800001u}, {0x80000000u, 0xbf800001u}};
    unsigned nt = std::max(1u, std::thread::hardware_concurrency());
    const uint32_t chunks = 512;
    struct Part {
        std::vector<uint32_t> k, v;
    };
    std::vector<Part> parts(2 * chunks);
    std::atomic<uint32_t> next(0);
    auto work = [&]() {
        for (;;) {
            uint32_t c = next.fetch_add(1);
            if (c >= 2 * chunks) break;
            uint32_t side = c / chunks, part = c % chunks;
            uint64_t lo = spans[side][0], hi = spans[side][1];
            uint64_t len = hi - lo;
            uint64_t a = lo + len * part / chunks, b = lo + len * (part + 1) / chunks;
            Part& P = parts[c];
            for (uint64_t u = a; u < b; u++) {
                float x = ffrom((uint32_t)u);
                float g = acosf(x);
                float r = (float)tpcf_acos_d((double)x);
                if (fbits(g) != fbits(r)) {
                    P.k.push_back((uint32_t)u);
                    P.v.push_back(fbits(g));
                }
            }
        }
    };
    std::vector<std::thread> th;
    for (unsigned t = 0; t < nt; t++) th.emplace_back(work);
    for (auto& t : th) t.join();
    AcosHost h;
    for (auto& P : parts) {
        h.keys.insert(h.keys.end(), P.k.begin(), P.k.end());
        h.vals.insert(h.vals.end(), P.v.begin(), P.v.end());
    }
    h.bucket.assign(65537, 0);
    size_t i = 0;
    for (uint32_t b = 0; b <= 65536; b++) {
        while (i < h.keys.size() && (h.keys[i] >> 16) < b) i++;
        h.bucket[b] = (uint32_t)i;
    }
    return h;
}

std::string acos_cache_path() {
    char name[256];
    // the table depends on the C library's acosf, the architecture and this
    // file's tpcf_acos_d; a probe value keys the latter
    uint32_t probe = fbits((float)tpcf_acos_d(0.3)) ^ fbits((float)tpcf_acos_d(-0.87));
#if defined(__aarch64__)
    const char* arch = "aarch64";
#elif defined(__x86_64__)
    const char* arch = "x86_64";
#else
    const char* arch = "other";
#endif
    snprintf(name, sizeof(name), "/acosf_exc_v1_%s_glibc%s_%08x.bin", arch, gnu_get_libc_version(), probe);
    return cache_dir() + name;
}

AcosHost load_or_build_acos_table() {
    std::string path = acos_cache_path();
    FILE* f = fopen(path.c_str(), "rb");
    if (f) {
        AcosHost h;
        uint32_t n = 0;
        bool ok = fread(&n, 4, 1, f) == 1 && n < (1u << 28);
        if (ok) {
            h.keys.resize(n);
            h.vals.resize(n);
            h.bucket.resize(65537);
            ok = fread(h.keys.data(), 4, n, f) == n && fread(h.vals.data(), 4, n, f) == n &&
                 fread(h.bucket.data(), 4, 65537, f) == 65537;
        }
        fclose(f);
        if (ok) return h;
    }
    AcosHost h = build_acos_table();
    mkdirs(cache_dir());
    std::string tmp = path + ".tmp" + std::to_string(getpid());
    f = fopen(tmp.c_str(), "wb");
    if (f) {
        uint32_t n = (uint32_t)h.keys.size();
        bool ok = fwrite(&n, 4, 1, f) == 1 && fwrite(h.keys.data(), 4, n, f) == n &&
                  fwrite(h.vals.data(), 4, n, f) == n && fwrite(h.bucket.data(), 4, 65537, f) == 65537;
        fclose(f);
        if (ok) rename(tmp.c_str(), path.c_str());
        else unlink(tmp.c_str());
    }
    return h;
}

// ---------------------------------------------------------------------------
// binning

struct Binning {
    int kind = 0;
    TriParams tri{};
    ThreeParams three{};
    NearParams near{};
    bool near_ok = false;     // three-side: the binning suits the neighbour lists
    bool list_ok = false;     // triangles: the same
    PairParams pair{};
    int len = 0;
    double lmax = INFINITY;   // no counted triangle/pair has a side >= lmax
    bool tri_prune = false;   // triangle: test the s and q ranges on tile-triple side bounds
    double s_lo = 0, s_hi = 0, q_hi = 0;
};

// Whether a job of this spec runs in the guarded FP32 kernels.  The fast
// triangle kernel keeps side words of 16 bits (s-bin below 255): binnings with
// more s bins are counted by the plain FP64 kernel, with the same histograms.
// The double-precision geometry takes the fast kernel where float sides and the
// guard bands tell its bins: coordinates of ordinary size (`tame`), a lower edge
// that a float separation cannot miss, bands well inside the bins.
bool guarded_fp32(const tpcf_spec& sp, const Binning& bin, bool tame) {
    if (sp.precision == TPCF_GEOMETRY_FP64)
        return tame && bin.tri.S <= MAX_FAST_S && (bin.tri.s_lo <= 0 || bin.tri.s_lo >= 1e-12f) &&
               bin.tri.geo_s_thr > 0.25f && bin.tri.q_thr > 0.25f && bin.tri.t_thrA > 0.25f;
    if (sp.precision != TPCF_GUARDED_FP32) return false;
    if (sp.kind == TPCF_TRIANGLE || sp.kind == TPCF_TRIANGLE_JBJ) return bin.tri.S <= MAX_FAST_S;
    return true;
}

float ref_bw(float lo, float hi, int n) {
    // (hist_max - hist_min)/nbins in float, as distance_to_bin computes it
    volatile float d = hi - lo;
    volatile float r = d / (float)n;
    return r;
}

// The three-side bin of a side whose squared length (as the reference sums
// it) is d2: distance_to_bin of src/3pcf_C_version.cc:23-51 on sqrtf(d2),
// nbins + 1 standing for d >= hist_max.  IEEE single operations, as on the
// device.
static int three_side_bin_of_d2(float d2, float lo, float hi, float bw, int n) {
    volatile float d = sqrtf(d2);
    if (d < lo) return 0;
    if (d >= hi) return n + 1;
    volatile float x = d - lo;
    volatile float q = x / bw;
    return (int)q;
}

// Thresholds u[v] (smallest float d2 >= 0 with bin >= v) by bisection over
// the ordered bit patterns of non-negative floats; the bin is a
// non-decreasing function of d2 (sqrt, subtraction, division and truncation
// all are).  Returns false where the first guess inv_bw * (sqrt(d2) - lo)
// might be off by more than one bin (very fine binnings).
static bool three_side_thresholds(ThreeParams& p) {
    if (p.n + 3 > TS_UMAX) return false;
    if (std::max(fabs((double)p.lo), fabs((double)p.hi)) / (double)p.bw > 16384.0) return false;
    p.inv_bw = 1.0f / p.bw;
    p.u[0] = -INFINITY;
    for (int v = 1; v <= p.n + 1; v++) {
        uint32_t lo = 0, hi = 0x7F800000u;  // +0 .. +inf (bin nbins + 1)
        while (lo < hi) {
            const uint32_t mid = lo + (hi - lo) / 2;
            float x;
            memcpy(&x, &mid, 4);
            if (three_side_bin_of_d2(x, p.lo, p.hi, p.bw, p.n) >= v) hi = mid;
            else lo = mid + 1;
        }
        memcpy(&p.u[v], &lo, 4);
    }
    p.u[p.n + 2] = NAN;
    for (int v = p.n + 3; v < TS_UMAX; v++) p.u[v] = NAN;
    return true;
}

Binning make_binning(const tpcf_spec& sp) {
    Binning b;
    b.kind = sp.kind;
    auto check_axis = [](const tpcf_axis& a, const char* what) {
        if (a.nbins <= 0 || a.nbins > 100000) throw InvalidArg{std::string("bad nbins for ") + what};
        if (!(a.hi > a.lo)) throw InvalidArg{std::string("need hi > lo for ") + what};
    };
    if (sp.kind == TPCF_THREE_SIDE) {
        check_axis(sp.axis[0], "three-side axis");
        ThreeParams& p = b.three;
        p.n = sp.axis[0].nbins;
        if ((int64_t)p.n * p.n * p.n > (1 << 29)) throw InvalidArg{"three-side nbins too large"};
        p.lo = sp.axis[0].lo;
        p.hi = sp.axis[0].hi;
        p.bw = ref_bw(p.lo, p.hi, p.n);
        p.clean = sp.overflow == TPCF_OVERFLOW_CLEAN;
        p.len = p.n * p.n * p.n;
        b.len = p.len;
        if (p.clean) b.lmax = (double)p.hi * (1 + 1e-6);
        // (compat mode counts every triple: the side codes are a small part of its work)
        p.fast = p.clean && three_side_thresholds(p) ? 1 : 0;
        p.zcode = three_side_bin_of_d2(0.0f, p.lo, p.hi, p.bw, p.n);
        PairParams g{};  // the same bins below hist_max
        g.n = p.n;
        g.lo = p.lo;
        g.hi = p.hi;
        g.bw = p.bw;
        pair_guard(g);
        const double r2 = (double)p.hi * (1 + 1e-6) * (double)p.hi;
        b.near = {p.n, p.len, p.clean, p.zcode, p.lo, p.hi, p.bw, g.inv_bw, g.off, g.thr,
                  nextafterf((float)std::min(r2, 3e38), INFINITY)};
        b.near_ok = sp.prune && sp.precision == TPCF_GUARDED_FP32 && g.fast && g.thr > 0.25f && p.hi > 0 && p.hi <= 1e15f;
    } else if (sp.kind == TPCF_TRIANGLE) {
        for (int a = 0; a < 3; a++) check_axis(sp.axis[a], "triangle axis");
        TriParams& p = b.tri;
        p.S = sp.axis[0].nbins;
        p.Q = sp.axis[1].nbins;
        p.T = sp.axis[2].nbins;
        if ((int64_t)p.S * p.Q * p.T > MAX_TRI_BINS) throw InvalidArg{"triangle binning too large"};
        p.len = p.S * p.Q * p.T;
        p.s_lo = sp.axis[0].lo;
        p.s_hi = sp.axis[0].hi;
        p.s_bw = ref_bw(p.s_lo, p.s_hi, p.S);
        p.q_lo = sp.axis[1].lo;
        p.q_hi = sp.axis[1].hi;
        p.q_bw = ref_bw(p.q_lo, p.q_hi, p.Q);
        p.t_lo = sp.axis[2].lo;
        p.t_hi = sp.axis[2].hi;
        p.t_bw = ref_bw(p.t_lo, p.t_hi, p.T);
        p.nan_zero = sp.nan_policy == TPCF_NAN_ZERO;
        // q coordinate: (q - q_lo)/q_bw; guard covers |fast - reference| <= ~9 ulp(q)/q_bw
        double qs = 1.0 / (double)p.q_bw;
        p.q_scale = (float)qs;
        p.q_off = (float)(-(double)p.q_lo * qs - 0.5);
        double qmax = std::max(fabs((double)p.q_lo), fabs((double)p.q_hi));
        p.q_thr = (float)(0.5 - (8e-7 * qmax * qs + 2e-6));
        // theta coordinate: acos(c)/(pi' t_bw) - t_lo/t_bw with pi' = 3.14159
        const double pi_ref = 3.14159, pi = 3.14159265358979323846;
        double K = 1.0 / (pi_ref * (double)p.t_bw);
        // acos(x) ~ sqrt(1 - x) * P(x) on [0, 1], P of degree 5: a minimax (Remez)
        // fit in absolute error, which equioscillates at 7 points with
        // |sqrt(1 - x) P(x) - acos(x)| <= 6.37e-7 rad (largest at x = 0; pinned
        // by tests/test_thresholds.py on a grid of 2e6 points).  The guard band
        // below budgets 6.4e-7 rad for it.
        static const double coef[6] = {1.5707956894727488, -0.2145428141209928, 0.08817102789580339,
                                       -0.0459271445289548, 0.020619951348088413, -0.004911124693855812};
        for (int i = 0; i < 6; i++) p.t_coef[i] = (float)(coef[i] * K);
        p.t_half = (float)(K * pi / 2);
        p.t_off0 = (float)(K * pi / 2 - (double)p.t_lo / (double)p.t_bw - 0.5);
        // fixed part: polynomial (6.4e-7 rad) + float evaluation + reference
        // acosf (<= 1.5 ulp) and roundings, bounded by 4e-6 rad; plus relative
        // rounding of the coordinate itself
        double tmax = std::max(fabs((double)p.t_lo), fabs((double)p.t_hi)) / (double)p.t_bw + K * pi;
        double A = 4e-6 * K + 1e-6 * tmax + 2e-6;
        p.t_thrA = (float)(0.5 - A);
        // c-dependent part: |dc| <= 7e-7 |c| (reciprocals of two sides, products, the
        // reference's roundings: 9 x 2^-24, and a margin) amplified by 1/sqrt(1-c^2) <= 1/sqrt(1-|c|)
        p.t_thrB = (float)(7e-7 * K);
        // A cosine that the reference rounds beyond +-1 gives it NaN, which has a bin
        // of its own or none.  Where the angles 0 and pi lie on bin edges, as with
        // [0, 1), the bands hold every such triangle; else the band takes in the
        // whole bin as the cosine comes within 7e-7 of +-1.
        auto at_edge = [&](double angle) {
            const double x = (angle / pi_ref - (double)p.t_lo) / (double)p.t_bw;
            return fabs(x - nearbyint(x)) <= 1e-4 * K;
        };
        if (!at_edge(0) || !at_edge(pi)) p.t_thrB = (float)std::max(7e-7 * K, 4.2e-4);
        p.t2_off = (float)((1.0 - 3.0 * (double)p.t_lo) / (double)p.t_bw - 1.5);
        p.theta_full = (p.t_lo <= 0.f && p.t_hi >= 1.f);
        if (sp.precision == TPCF_GEOMETRY_FP64) {
            // the guard bands of the geometry (triangle_full2): relative errors of
            // 4e-7 of a side, 3e-6 of a ratio, and of the coordinates themselves
            p.geo_s_below = p.s_lo > 0 ? (float)std::max(1e-15, (double)p.s_lo * (1 - 1e-6)) : -1.f;
            p.geo_s_above = (float)((double)p.s_hi * (p.s_hi > 0 ? 1 + 1e-6 : 1 - 1e-6));
            const double smax = std::max(fabs((double)p.s_lo), fabs((double)p.s_hi)) / (double)p.s_bw;
            p.geo_s_inv = (float)(1.0 / (double)p.s_bw);
            p.geo_s_off = (float)(-(double)p.s_lo / (double)p.s_bw - 0.5);
            p.geo_s_thr = (float)(0.5 - (2e-6 * smax + 1e-5));
            p.q_thr = (float)(0.5 - (3e-6 * qmax * qs + 1e-5));
            p.t_thrA = (float)(0.5 - (4e-6 * K + 2e-6 * tmax + 1e-5));
            p.geo_t = (float)(6e-6 * K);
        }
        b.len = p.len;
        // every counted permutation needs shortest or middle side < s_hi and a
        // ratio < q_hi; all sides are then below s_hi (1 + q_hi)
        if (p.s_hi > 0 && p.q_hi > 0) b.lmax = (double)p.s_hi * (1.0 + (double)p.q_hi) * (1 + 1e-5) + 1e-6;
        b.tri_prune = true;
        b.s_lo = p.s_lo;
        b.s_hi = p.s_hi;
        b.q_hi = (double)p.q_hi * (1 + 1e-5);
    } else if (sp.kind == TPCF_TRIANGLE_JBJ) {
        for (int a = 0; a < 3; a++) check_axis(sp.axis[a], "JBJ axis");
        TriParams& p = b.tri;
        p.S = sp.axis[0].nbins;
        p.Q = sp.axis[1].nbins;
        p.T = sp.axis[2].nbins;
        if ((int64_t)p.S * p.Q * p.T > MAX_TRI_BINS) throw InvalidArg{"JBJ binning too large"};
        p.len = p.S * p.Q * p.T;
        p.s_lo = sp.axis[0].lo;
        p.s_hi = sp.axis[0].hi;
        p.s_bw = ref_bw(p.s_lo, p.s_hi, p.S);
        p.q_lo = sp.axis[1].lo;
        p.q_hi = sp.axis[1].hi;
        p.q_bw = ref_bw(p.q_lo, p.q_hi, p.Q);
        p.t_lo = sp.axis[2].lo;
        p.t_hi = sp.axis[2].hi;
        p.t_bw = ref_bw(p.t_lo, p.t_hi, p.T);
        p.nan_zero = 0;  // no NaN reaches a counted JBJ bin (zero sides are dropped)
        // guard bands of the fast bins (jbj_full2); binnings too fine for them
        // take the reference's divisions for every triangle
        auto axis_guard = [](float lo, float hi, float bw, float& scale, float& off, float& thr) {
            const double D = std::max(fabs((double)lo), fabs((double)hi)) / (double)bw + 1.0;
            const bool ok = D <= 65536.0 && bw >= 1e-30f;
            scale = ok ? (float)(1.0 / (double)bw) : 1.0f;
            off = ok ? (float)(-(double)lo / (double)bw - 0.5) : 0.0f;
            thr = ok ? (float)(0.5 - 1e-6 * (D + 1.0)) : -1.0f;
        };
        axis_guard(p.q_lo, p.q_hi, p.q_bw, p.q_scale, p.q_off, p.q_thr);
        axis_guard(p.t_lo, p.t_hi, p.t_bw, p.t_coef[0], p.t_off0, p.t_thrA);
        b.len = p.len;
        // counted: s < s_hi, s/m >= q_lo, (l - m)/s < t_hi, so
        // l < s_hi/q_lo + max(t_hi, 0) s_hi (margins cover the float roundings)
        if (p.q_lo > 0 && p.s_hi > 0)
            b.lmax = ((double)p.s_hi / (double)p.q_lo + std::max(0.0, (double)p.t_hi) * (double)p.s_hi) * (1 + 1e-5) +
                     1e-6;
    } else if (sp.kind == TPCF_PAIR) {
        check_axis(sp.axis[0], "pair axis");
        PairParams& p = b.pair;
        p.n = sp.axis[0].nbins;
        p.lo = sp.axis[0].lo;
        p.hi = sp.axis[0].hi;
        p.bw = ref_bw(p.lo, p.hi, p.n);
        pair_guard(p);
        b.len = p.n;
        b.lmax = (double)p.hi * (1 + 1e-6) + 1e-6;
    } else {
        throw InvalidArg{"unknown kind"};
    }
    if (!sp.prune) {
        b.lmax = INFINITY;
        b.tri_prune = false;
    }
    if (sp.kind == TPCF_PAIR) {
        const double r2 = b.lmax * b.lmax;
        // (no counted separation at all below a negative upper edge)
        b.pair.reach2 = b.lmax < 0 ? 0.f : r2 < 3e38 ? nextafterf((float)r2, INFINITY) : INFINITY;
    }
    if (sp.kind == TPCF_TRIANGLE || sp.kind == TPCF_TRIANGLE_JBJ) {
        // a counted triangle has its shortest side below s_hi and its middle one
        // below q_hi S or s_hi (JBJ: at most S / q_lo); margins cover the roundings
        TriParams& p = b.tri;
        const bool jbj = sp.kind == TPCF_TRIANGLE_JBJ;
        const double q = jbj ? (p.q_lo > 0 ? 1.0 / (double)p.q_lo : INFINITY) : (double)p.q_hi;
        const double reach = std::max((double)p.s_hi * q, jbj ? 0.0 : (double)p.s_hi) * (1 + 2e-5) + 1e-6;
        b.list_ok = sp.prune && p.s_hi > 0 && q > 0 && reach < 1e15 && p.S <= MAX_FAST_S;
        if (b.list_ok) {
            p.list_r2 = nextafterf((float)(reach * reach), INFINITY);
            p.list_q = nextafterf((float)(q * (1 + 1e-5)), INFINITY);
            // guard bands of tri_list_bin
            const double K = 1.0 / (3.14159 * (double)p.t_bw);
            const double qmax = std::max(fabs((double)p.q_lo), fabs((double)p.q_hi)) / (double)p.q_bw;
            const bool geo = sp.precision == TPCF_GEOMETRY_FP64;
            p.list_t = jbj ? (float)(1e-6 / (double)p.t_bw) : (float)((geo ? 6e-6 : 2.2e-6) * K);
            p.list_q_thr = geo ? p.q_thr : (float)(0.5 - (1.2e-6 * qmax + 3e-6));
            p.list_top = jbj ? 0.f : nextafterf((float)((double)p.s_hi * (1 + 1e-5)), INFINITY);
        }
    }
    // device copy of the bound, rounded up so that a float side >= it is >= lmax
    if (sp.kind == TPCF_TRIANGLE || sp.kind == TPCF_TRIANGLE_JBJ) {
        TriParams& p = b.tri;
        p.lmax = b.lmax < 3e38 ? nextafterf((float)b.lmax, INFINITY) : INFINITY;
        const double q = sp.kind == TPCF_TRIANGLE ? (double)p.q_hi : p.q_lo > 0 ? 1.0 / (double)p.q_lo : 0.0;
        auto limit = [&](double side) {
            const double mid = side * q * (1 + 1e-5) + 1e-6;
            return sp.prune && q > 0 && mid < 3e38 ? nextafterf((float)mid, INFINITY) : INFINITY;
        };
        p.mid_hi = limit((double)p.s_hi);
        // the split lets the fewest triangles through to the binning on
        // clustered data (77 to 83 % for splits at 0.6 to 0.8 of s_hi; of the
        // benchmark's binning -- other binnings take the same, JBJ included, where
        // another share might let fewer through)
        p.s_split = std::max(p.s_lo, 0.72f * p.s_hi);
        p.mid_split = std::max(p.s_hi, limit((double)p.s_split));
    }
    return b;
}

bool same_binning(const tpcf_spec& a, const tpcf_spec& b) {
    if (a.kind != b.kind || a.precision != b.precision) return false;
    if (a.kind == TPCF_TRIANGLE && a.nan_policy != b.nan_policy) return false;
    if ((a.kind == TPCF_THREE_SIDE || a.kind == TPCF_TRIANGLE_JBJ) && a.overflow != b.overflow) return false;
    int na = (a.kind == TPCF_TRIANGLE || a.kind == TPCF_TRIANGLE_JBJ) ? 3 : 1;
    for (int i = 0; i < na; i++)
        if (a.axis[i].lo != b.axis[i].lo || a.axis[i].hi != b.axis[i].hi || a.axis[i].nbins != b.axis[i].nbins)
            return false;
    return true;
}

// ---------------------------------------------------------------------------
// loop units (the reference's numcalc / fake_tot)

uint64_t loop_units(int kind, int loop, const int64_t n[3]) {
    if (kind == TPCF_THREE_SIDE || (kind != TPCF_PAIR && loop == TPCF_LOOP_ALL)) return (uint64_t)n[0] * n[1] * n[2];
    if (kind == TPCF_PAIR && loop != TPCF_LOOP_SAME) return (uint64_t)n[0] * n[1];
    // Sums of the loops' bounds in closed form, modulo 2^64.  (A range whose end
    // lies before its begin has a negative size: its loop does not run.)
    const uint64_t last = kind == TPCF_PAIR ? n[1] : n[2];
    const int64_t outer = kind == TPCF_PAIR ? std::min(n[0], n[1]) : std::min(n[1], n[2]);
    if (outer <= 0) return 0;
    const uint64_t m = outer, tail = m * last - m * (m - 1) / 2;  // sum over j < m of last - j
    if (kind == TPCF_PAIR) return tail;
    const uint64_t n0 = n[0];
    if (loop == TPCF_LOOP_ONE) return n0 * tail;
    // LOOP_SAME: min(n0, j + 1) points i for each j
    const uint64_t p = n[0] > 0 ? std::min(m, n0) : 0;
    const uint64_t lin = p ? p * (p - 1) / 2 : 0;                                  // sums of j and j^2 over j < p
    const uint64_t sq = lin % 3 == 0 ? lin / 3 * (2 * p - 1) : lin * ((2 * p - 1) / 3);
    const uint64_t head = p * last + last * lin - lin - sq;                        // (j + 1) (last - j)
    return head + n0 * (tail - (p * last - lin));
}

// ---------------------------------------------------------------------------
// context

// One lane = one stream with its own scratch buffers.  The synchronous API uses
// lane 0; every serving worker owns one further lane, so batches of different
// workers run concurrently on the device.
struct Lane {
    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr, ev_mid = nullptr;
    uint64_t h2d = 0, d2h = 0;  // bytes copied since the last stats read
    DevBuf<DevJob> d_jobs;
    PinnedBuf<DevJob> h_jobs;         // device jobs of the batch being planned
    PinnedBuf<uint32_t> h_rows;
    DevBuf<uint32_t> d_rows;          // first row (pairs: item) of each job, and the end
    DevBuf<uint2> d_row_cnt, d_block_sum;
    DevBuf<uint4> d_units;            // the plan: units and their A tiles
    DevBuf<uint32_t> d_masks;
    DevBuf<unsigned int> d_counters;  // see CTR_*
    DevBuf<uint4> d_queue;
    DevBuf<unsigned long long> d_hist;
    DevBuf<unsigned long long> d_acc;  // three-side accumulators of the neighbour lists
    PinnedBuf<unsigned long long> h_hist;
    PinnedBuf<unsigned int> h_counters;
    // last planned batch (see run_group)
    std::vector<uint64_t> plan_sig;
    uint32_t plan_rows = 0;  // rows (pairs: items) of the plan
    int plan_chunk = 0;      // pairs: tiles B per item; neighbour lists: centres per item
    int plan_parts = 1, plan_kparts = 1;  // triangle lists: shares of a centre
    uint32_t plan_wedges = 0;  // neighbour lists: items of the wedge kernel
    // the launch sequence of the last batch, captured as a CUDA graph and
    // replayed while the batch and every buffer it touches stay the same
    cudaGraphExec_t graph = nullptr;
    std::vector<uint64_t> graph_sig;
    bool graphs_ok = true;
    // SMs a launch of this lane may fill with its persistent CTAs (0: all);
    // the serving lane that runs heavy jobs leaves some to the light lanes
    int sm_cap = 0;
    // count in slices of the task list (heavy serving batches)
    bool slice_batches = false;
    tpcf_stats stats{};
    void drop_graph() {
        if (graph) cudaGraphExecDestroy(graph);
        graph = nullptr;
        graph_sig.clear();
    }
    void release() {
        drop_graph();
        h_hist.release();
        h_counters.release();
        d_jobs.release();
        h_jobs.release();
        h_rows.release();
        d_rows.release();
        d_row_cnt.release();
        d_block_sum.release();
        d_units.release();
        d_masks.release();
        d_counters.release();
        d_queue.release();
        d_hist.release();
        d_acc.release();
        if (ev0) cudaEventDestroy(ev0);
        if (ev1) cudaEventDestroy(ev1);
        if (ev_mid) cudaEventDestroy(ev_mid);
        if (stream) cudaStreamDestroy(stream);
        ev0 = ev1 = ev_mid = nullptr;
        stream = nullptr;
    }
};

// shares of centres per warp of the triangle lists at least
constexpr uint64_t TL_WANT = 32;

// d_counters: words zeroed before every count, then the header of the plan
constexpr int CTR_WORK = 0;     // units (items) handed out
constexpr int CTR_RECHECK = 1;  // queued guard-band triangles
constexpr int CTR_EVAL = 2;     // evaluated (two words), binned (pairs: tile pairs; two words)
constexpr int CTR_DENSE = 6;    // neighbour lists: a centre has too many near tiles
constexpr int CTR_ZEROED = 8;
constexpr int CTR_HEADER = 8;
constexpr int CTR_WORDS = CTR_HEADER + (int)(sizeof(PlanHeader) / sizeof(unsigned int));

struct Pending {
    uint64_t ticket;
    double t_submit = 0, t_start = 0, t_done = 0;  // steady-clock ms
    double cost = 0;                                // job_cost at submission
    tpcf_spec spec;
    tpcf_job job;
    std::vector<uint64_t> result;
    tpcf_status status = 1;  // 1 = pending
    bool cancelled = false;
};

struct GroupJob {
    const tpcf_spec* spec;
    const tpcf_job* job;
    uint64_t* out;
    bool accumulate = false;  // add into out (jobs sharing out share one device histogram)
};

// A tiles [begin, end) of a group of one job (end < 0: all)
struct TileRange {
    int begin = 0, end = -1;
};

// Thrown by run_group, before anything is counted, where a group's plan passes
// its limits (see count_group); tiles: A tiles of its first job; lists: it was to
// be counted from neighbour lists.
struct TooLarge {
    int tiles;
    bool lists;
};

// The limits of one plan: its units (21 GB of unit list), its rows (4 GB of
// counts a row) or items.  TPCF_MAX_UNITS, TPCF_MAX_ROWS: lower ones (tests use
// them to have small batches counted in parts).
uint32_t plan_limit(const char* env, uint32_t most) {
    const char* e = getenv(env);
    return e ? (uint32_t)std::min<long>(std::max(1L, std::atol(e)), most) : most;
}
constexpr uint32_t MAX_UNITS = 1u << 30, MAX_ROWS = 1u << 29, MAX_ITEMS = 0xF0000000u;

}  // namespace

// Launch shape of a persistent kernel: warp-private histogram copies in
// shared memory (0: count straight into the 64-bit global histogram),
// resident CTAs per SM (the grid is that many per SM) and, for the
// three-side kernel, task pipelines per CTA (0: plain 8-warp CTAs; g > 0:
// one CTA per SM of g 8-warp pipelines around one large histogram).
struct Shape {
    int copies = 1;
    int per_sm = 1;
    int groups = 0;
    size_t smem = 0;
};

struct tpcf_ctx {
    int device = 0;
    int num_sms = 0;
    int max_smem_sm = 0, max_smem_block = 0;  // shared memory of an SM, most of a block
    std::recursive_mutex mu;      // serialises the synchronous API (lane 0)
    std::recursive_mutex view_mu; // catalogs and spatial views
    std::mutex acos_mu;
    std::string last_error;
    uint64_t next_handle = 1;
    std::map<uint64_t, std::shared_ptr<Catalog>> catalogs;
    // (catalog, begin, end, tile points, global loop indices) -> view
    std::map<std::tuple<uint64_t, int64_t, int64_t, int, bool>, std::shared_ptr<View>> views;
    // full views of new catalogs being built in the background
    struct PendingView {
        std::shared_future<std::shared_ptr<View>> fut;
        uint64_t id;
        int64_t n;
    };
    std::map<std::tuple<uint64_t, int64_t, int64_t, int, bool>, PendingView> pending_views;
    int tile_points = TILE;  // points per spatial tile (<= TILE)
    uint64_t next_view_id = 0;
    // acos table
    bool acos_ready = false;
    DevBuf<uint32_t> acos_keys, acos_vals, acos_bucket;
    uint32_t acos_n = 0;
    std::vector<std::unique_ptr<Lane>> lanes;
    // serving
    std::mutex qmu;
    std::condition_variable qcv;
    std::deque<std::shared_ptr<Pending>> queue;
    std::map<uint64_t, std::shared_ptr<Pending>> tickets;
    uint64_t next_ticket = 1;
    std::vector<std::thread> workers;
    bool stop = false;
    // serving trace (TPCF_SERVING_TRACE=file): one line per batch, written by
    // tpcf_destroy: lane, jobs, first ticket, oldest submit, start, planned, done (ms)
    std::string trace_path;
    std::vector<std::string> trace;
    int64_t admit_bytes = (int64_t)8 << 30;
    double heavy_cost = 4e11;  // job_cost above which a job runs alone on the first serving lane (~50 ms)
    double light_batch_cost = 1e11;  // summed job_cost at which a batch of light jobs closes
    std::map<std::tuple<uint64_t, int64_t, int64_t, uint64_t, int64_t, int64_t, double>, double> density;
    int reserve_sms = 0;       // SMs a heavy serving batch leaves free for light jobs
    bool slice_heavy = true;   // heavy serving batches count in slices (light lanes run between them)
    int slice_tasks = 0;       // tasks per slice (0: at least 8 per CTA and at most 64 slices)
    int group_tasks = 0;       // A tiles per row of the planner, sharing one j-k table (0: by the batch)
    int64_t inflight_bytes = 0;  // device bytes of batches running on serving lanes
    // share of the pairs of two catalog ranges within a reach (see pair_share; under view_mu)
    std::map<std::tuple<uint64_t, int64_t, int64_t, uint64_t, int64_t, int64_t, float>, double> shares;
    // autotuner: launch shape per batch signature, and the batches whose
    // neighbour lists the device refused (counted from tiles)
    std::mutex tune_mu;
    std::map<uint64_t, Shape> tuned;
    std::unordered_set<uint64_t> refused;
};

namespace {

tpcf_status fail(tpcf_ctx* ctx, tpcf_status s, const std::string& msg) {
    if (ctx) ctx->last_error = msg;
    g_tls_error = msg;
    return s;
}

// TPCF_PLAN_TRACE=1: wall times of view building and batch planning on stderr
bool plan_trace() {
    static const bool on = [] {
        const char* e = getenv("TPCF_PLAN_TRACE");
        return e && e[0] == '1';
    }();
    return on;
}

// Builds the spatial view of points [begin, end) of a catalog: k-d order,
// tiles, their boxes, and the device copy (on stream st, synchronized).
std::shared_ptr<View> build_view(const Catalog& c, int64_t begin, int64_t end, int tile, bool global, uint64_t id,
                                 cudaStream_t st) {
    const auto tv0 = std::chrono::steady_clock::now();
    auto v = std::make_shared<View>();
    v->id = id;
    int64_t n = end - begin;
    v->n = n;
    std::vector<float> xyz(3 * (size_t)n);
    for (int64_t i = 0; i < n; i++) {
        xyz[3 * i] = c.x[begin + i];
        xyz[3 * i + 1] = c.y[begin + i];
        xyz[3 * i + 2] = c.z[begin + i];
    }
    std::vector<int32_t> order(n);
    std::iota(order.begin(), order.end(), 0);
    const auto tv1 = std::chrono::steady_clock::now();
    kd_order(xyz.data(), order, n, tile);
    const auto tv2 = std::chrono::steady_clock::now();
    v->ntiles = (int)((n + tile - 1) / tile);
    std::vector<float4> pts(std::max<int64_t>(n, 1));
    for (int64_t i = 0; i < n; i++) {
        int32_t o = order[i];
        float4 p;
        p.x = xyz[3 * (size_t)o];
        p.y = xyz[3 * (size_t)o + 1];
        p.z = xyz[3 * (size_t)o + 2];
        // loop index inside the range, or inside the whole catalog
        int32_t key_i = global ? (int32_t)(o + begin) : o;
        memcpy(&p.w, &key_i, 4);
        pts[i] = p;
    }
    v->h_tile_start.resize(v->ntiles + 1);
    v->boxes.resize(v->ntiles);
    for (int t = 0; t <= v->ntiles; t++) v->h_tile_start[t] = (int32_t)std::min<int64_t>((int64_t)t * tile, n);
    for (int t = 0; t < v->ntiles; t++) {
        Box b;
        for (int a = 0; a < 3; a++) {
            b.lo[a] = INFINITY;
            b.hi[a] = -INFINITY;
        }
        for (int i = v->h_tile_start[t]; i < v->h_tile_start[t + 1]; i++) {
            const float* q = &pts[i].x;
            for (int a = 0; a < 3; a++) {
                b.lo[a] = std::min(b.lo[a], q[a]);
                b.hi[a] = std::max(b.hi[a], q[a]);
            }
        }
        v->boxes[t] = b;
    }
    for (const Box& b : v->boxes) {
        double w = 0;
        for (int a = 0; a < 3; a++) w = std::max(w, (double)b.hi[a] - (double)b.lo[a]);
        v->extent += w / v->ntiles;
    }
    const auto tv3 = std::chrono::steady_clock::now();
    v->pts.reserve(pts.size());
    CK(cudaMemcpyAsync(v->pts.p, pts.data(), pts.size() * sizeof(float4), cudaMemcpyHostToDevice, st));
    v->tile_start.reserve(v->ntiles + 1);
    CK(cudaMemcpyAsync(v->tile_start.p, v->h_tile_start.data(), (v->ntiles + 1) * sizeof(int32_t),
                       cudaMemcpyHostToDevice, st));
    std::vector<float4> dbox(2 * std::max<size_t>(v->boxes.size(), 1));
    for (size_t t = 0; t < v->boxes.size(); t++) {
        const Box& b = v->boxes[t];
        dbox[2 * t] = make_float4(b.lo[0], b.lo[1], b.lo[2], 0.f);
        dbox[2 * t + 1] = make_float4(b.hi[0], b.hi[1], b.hi[2], 0.f);
    }
    v->box.reserve(dbox.size());
    CK(cudaMemcpyAsync(v->box.p, dbox.data(), dbox.size() * sizeof(float4), cudaMemcpyHostToDevice, st));
    CK(cudaStreamSynchronize(st));
    v->upload_bytes = pts.size() * sizeof(float4) + (v->ntiles + 1) * sizeof(int32_t) + dbox.size() * sizeof(float4);
    if (plan_trace()) {
        auto ms = [](std::chrono::steady_clock::time_point a, std::chrono::steady_clock::time_point b) {
            return std::chrono::duration<double, std::milli>(b - a).count();
        };
        const auto tv4 = std::chrono::steady_clock::now();
        fprintf(stderr, "tpcf view: points %lld copy %.4f order %.4f pack %.4f upload %.4f\n", (long long)n,
                ms(tv0, tv1), ms(tv1, tv2), ms(tv2, tv3), ms(tv3, tv4));
    }
    return v;
}

// Id and point count of the view of catalog `handle` over [begin, end): a
// view being built in the background is not waited for (its id was assigned
// when it was started); any other is made now.
struct ViewRef {
    uint64_t id;
    int64_t n;
};

// The view of catalog `handle` over [begin, end) for the context's tile size:
// cached, being built in the background (a new catalog's full view), or built
// now on the lane's stream.  With ref != nullptr and the view still being
// built, returns nullptr at once and fills ref.
std::shared_ptr<View> get_view(tpcf_ctx* ctx, Lane& L, uint64_t handle, int64_t begin, int64_t end,
                               bool global = false, ViewRef* ref = nullptr) {
    std::unique_lock<std::recursive_mutex> vlk(ctx->view_mu);
    auto it = ctx->catalogs.find(handle);
    if (it == ctx->catalogs.end()) throw InvalidArg{"unknown catalog handle"};
    const std::shared_ptr<Catalog> cat = it->second;
    if (end < 0) end = cat->n;
    if (begin < 0 || begin > end || end > cat->n) throw InvalidArg{"catalog range out of bounds"};
    const int tile = ctx->tile_points;
    if (begin == 0) global = false;  // the same loop indices
    auto key = std::make_tuple(handle, begin, end, tile, global);
    auto vi = ctx->views.find(key);
    if (vi != ctx->views.end()) {
        if (ref) *ref = {vi->second->id, vi->second->n};
        return vi->second;
    }
    auto pi = ctx->pending_views.find(key);
    if (pi != ctx->pending_views.end()) {
        if (ref) {
            *ref = {pi->second.id, pi->second.n};
            return nullptr;
        }
        std::shared_future<std::shared_ptr<View>> fut = pi->second.fut;
        vlk.unlock();
        std::shared_ptr<View> v;
        try {
            v = fut.get();
        } catch (...) {
            vlk.lock();
            ctx->pending_views.erase(key);
            throw;
        }
        vlk.lock();
        ctx->pending_views.erase(key);
        if (!ctx->catalogs.count(handle)) throw InvalidArg{"unknown catalog handle"};
        auto ins = ctx->views.emplace(key, v);
        if (ins.second) L.h2d += v->upload_bytes;
        return ins.first->second;
    }
    auto v = build_view(*cat, begin, end, tile, global, ++ctx->next_view_id, L.stream);
    L.h2d += v->upload_bytes;
    ctx->views[key] = v;
    if (ref) *ref = {v->id, v->n};
    return v;
}

void ensure_acos(tpcf_ctx* ctx) {
    std::lock_guard<std::mutex> alk(ctx->acos_mu);
    if (ctx->acos_ready) return;
    AcosHost h = load_or_build_acos_table();
    ctx->acos_n = (uint32_t)h.keys.size();
    ctx->acos_keys.reserve(std::max<size_t>(h.keys.size(), 1));
    ctx->acos_vals.reserve(std::max<size_t>(h.vals.size(), 1));
    ctx->acos_bucket.reserve(65537);
    if (!h.keys.empty()) {
        CK(cudaMemcpy(ctx->acos_keys.p, h.keys.data(), h.keys.size() * 4, cudaMemcpyHostToDevice));
        CK(cudaMemcpy(ctx->acos_vals.p, h.vals.data(), h.vals.size() * 4, cudaMemcpyHostToDevice));
    }
    CK(cudaMemcpy(ctx->acos_bucket.p, h.bucket.data(), 65537 * 4, cudaMemcpyHostToDevice));
    ctx->acos_ready = true;
}

AcosTable acos_table(tpcf_ctx* ctx) {
    AcosTable t;
    t.keys = ctx->acos_keys.p;
    t.vals = ctx->acos_vals.p;
    t.bucket = ctx->acos_bucket.p;
    t.n = ctx->acos_n;
    return t;
}

// Host worker threads for building views, started once per process (thread
// creation would cost more than a small view).  run() calls fn(i) for i in
// [0, n) on the workers and the calling thread; a run that finds the pool busy
// does its items inline.
class HostPool {
  public:
    static HostPool& get() {
        static HostPool pool;
        return pool;
    }
    // Runs fn(0..n) on this thread and the pool's threads.  Several callers
    // (a count's planning, background view builds, serving lanes) share the
    // pool: idle threads help whichever jobs have items left.
    void run(size_t n, const std::function<void(size_t)>& fn) {
        if (n == 0) return;
        if (workers_.empty() || n == 1) {
            for (size_t i = 0; i < n; i++) fn(i);
            return;
        }
        Job job;
        job.fn = &fn;
        job.n = n;
        {
            std::lock_guard<std::mutex> lk(mu_);
            jobs_.push_back(&job);
            posted_.fetch_add(1);
        }
        cv_.notify_all();
        try {
            work(job);
        } catch (...) {
            // no further items; wait for the helpers to leave the job (it lives
            // on this frame) before the exception leaves it
            job.next.store(n);
            std::unique_lock<std::mutex> lk(mu_);
            jobs_.erase(std::find(jobs_.begin(), jobs_.end(), &job));
            done_cv_.wait(lk, [&] { return job.users == 0; });
            throw;
        }
        std::unique_lock<std::mutex> lk(mu_);
        jobs_.erase(std::find(jobs_.begin(), jobs_.end(), &job));  // no new helpers
        done_cv_.wait(lk, [&] { return job.users == 0 && job.done.load() == n; });
    }
    ~HostPool() {
        {
            std::lock_guard<std::mutex> lk(mu_);
            stop_ = true;
            stop_flag_.store(true);
        }
        cv_.notify_all();
        for (auto& t : workers_) t.join();
    }

  private:
    struct Job {
        const std::function<void(size_t)>* fn = nullptr;
        size_t n = 0;
        std::atomic<size_t> next{0}, done{0};
        size_t users = 0;  // pool threads working on it (under mu_)
    };
    HostPool() {
        const unsigned n = std::max(1u, std::thread::hardware_concurrency()) - 1;
        for (unsigned t = 0; t < n; t++) workers_.emplace_back([this] { loop(); });
    }
    void work(Job& j) {
        for (;;) {
            size_t i = j.next.fetch_add(1);
            if (i >= j.n) break;
            (*j.fn)(i);
            j.done.fetch_add(1);
        }
    }
    Job* open_job() {  // under mu_
        for (Job* j : jobs_)
            if (j->next.load() < j->n) return j;
        return nullptr;
    }
    void loop() {
        uint64_t seen = 0;
        for (;;) {
            // the phases of a planning pass follow one another within
            // microseconds: watch for the next job for a while before sleeping
            // (a wake-up from the condition variable costs tens of microseconds)
            const auto spin_end = std::chrono::steady_clock::now() + std::chrono::microseconds(300);
            while (posted_.load() == seen && !stop_flag_.load() && std::chrono::steady_clock::now() < spin_end)
                std::this_thread::yield();
            Job* j = nullptr;
            {
                std::unique_lock<std::mutex> lk(mu_);
                cv_.wait(lk, [&] { return stop_ || (j = open_job()) != nullptr || posted_.load() != seen; });
                if (stop_) return;
                seen = posted_.load();
                if (!j) j = open_job();
                if (!j) continue;
                j->users++;
            }
            work(*j);
            {
                std::lock_guard<std::mutex> lk(mu_);
                j->users--;
            }
            done_cv_.notify_all();
        }
    }
    std::mutex mu_;
    std::condition_variable cv_, done_cv_;
    std::vector<std::thread> workers_;
    std::vector<Job*> jobs_;
    std::atomic<uint64_t> posted_{0};  // jobs posted so far
    std::atomic<bool> stop_flag_{false};
    bool stop_ = false;
};

void parallel_items(size_t n, const std::function<void(size_t)>& fn) { HostPool::get().run(n, fn); }

size_t shape_smem(const tpcf_spec& sp, const Binning& bin, int copies, int groups) {
    if (sp.kind == TPCF_TRIANGLE || sp.kind == TPCF_TRIANGLE_JBJ) return triangle_smem_bytes(bin.len, copies, sp.kind == TPCF_TRIANGLE_JBJ);
    if (sp.kind == TPCF_THREE_SIDE) return three_side_smem_bytes(bin.three, copies, groups);
    return pair_smem_bytes(bin.len, copies);
}

// Launch shapes worth trying for a group, the default first.  The guarded
// triangle kernel is compiled for four CTAs per SM (its register budget);
// the others take as many CTAs as shared memory allows, up to 8.
std::vector<Shape> shape_candidates(tpcf_ctx* ctx, const tpcf_spec& sp, const Binning& bin, bool fp64, bool near, int tlist) {
    const int max_smem_sm = ctx->max_smem_sm, max_smem_block = ctx->max_smem_block;
    auto fit = [&](int copies, int cap_per_sm, int groups = 0) {
        Shape sh;
        sh.copies = copies;
        sh.groups = groups;
        sh.smem = shape_smem(sp, bin, copies, groups);
        sh.per_sm = 0;
        if (sh.smem + 1024 > (size_t)max_smem_block) return sh;  // leaves room for the kernels' static shared memory
        sh.per_sm = std::min(cap_per_sm, (int)(max_smem_sm / (sh.smem + 1024)));
        return sh;
    };
    std::vector<Shape> out;
    auto add = [&](Shape sh) {
        if (sh.per_sm < 1) return;
        for (const Shape& o : out)
            if (o.copies == sh.copies && o.per_sm == sh.per_sm && o.groups == sh.groups) return;
        out.push_back(sh);
    };
    if (near) {  // one CTA per SM of up to four pipelines
        for (int g : {4, 2, 1}) {
            Shape sh;
            sh.groups = g;
            sh.smem = three_near_smem_bytes(bin.three.n, g);
            sh.per_sm = sh.smem + 1024 <= (size_t)max_smem_block ? 1 : 0;
            add(sh);
        }
        return out;
    }
    if (tlist) {  // (tlist: output slots of the launch)
        // as many warps per SM as the registers and the lists' shared memory
        // allow, in CTAs of 8 to 24 warps that share histograms; groups: warps per CTA
        for (int w : {8, 24, 12, 20, 16}) {
            Shape sh;
            sh.groups = w;
            // every slot's histogram in shared memory where they take at most 24 KB of a CTA
            sh.copies = (size_t)bin.len * 4 * tlist <= 24576 ? tlist : 1;
            sh.smem = tri_list_smem_bytes(bin.len, sh.copies, w);
            sh.per_sm = sh.smem + 1024 <= (size_t)max_smem_block
                            ? std::min(TL_MAX_WARPS / w, (int)(max_smem_sm / (sh.smem + 1024))) : 0;
            add(sh);
        }
        std::stable_sort(out.begin(), out.end(),
                         [](const Shape& a, const Shape& b) { return a.per_sm * a.groups > b.per_sm * b.groups; });
        if (out.size() > 3) out.resize(3);
        return out;
    }
    if (sp.kind == TPCF_TRIANGLE || sp.kind == TPCF_TRIANGLE_JBJ) {
        const char* bps = getenv("TPCF_TRI_BLOCKS_PER_SM");
        const int tri_per_sm = fp64 ? 2 : (bps ? std::max(1, atoi(bps)) : 4);
        // default: as many copies as keep four CTAs on an SM (the kernel
        // needs the warps to hide the latency of its shared-memory tables);
        // the autotuner also tries three CTAs with more copies
        int c = 8;
        while (c > 1 && fit(c, tri_per_sm).per_sm < tri_per_sm) c /= 2;
        add(fit(c, tri_per_sm));
        if (!fp64) {
            for (int cc : {4, 2, 1}) add(fit(cc, tri_per_sm));
            if (!bps)
                for (int cc : {4, 2, 1}) add(fit(cc, 3));
        }
        if (out.empty()) throw InvalidArg{"triangle histogram too large for shared memory"};
    } else if (sp.kind == TPCF_THREE_SIDE) {
        // default: the most copies that still leave four 8-warp CTAs per SM,
        // else one CTA per SM of as many pipelines (up to four) as fit
        // around one shared histogram, else the global histogram
        Shape def;
        def.copies = -1;
        for (int cc : {4, 2, 1}) {
            Shape sh = fit(cc, 8);
            if (sh.per_sm >= 4) {
                def = sh;
                break;
            }
        }
        int groups = 4;
        while (groups > 1 && fit(1, 1, groups).per_sm < 1) groups--;
        if (def.copies < 0) def = fit(1, 1, groups);
        if (def.per_sm < 1) def = fit(0, 8);
        add(def);
        for (int cc : {8, 4, 2, 1, 0}) add(fit(cc, 8));
        add(fit(1, 1, groups));
    } else {
        Shape def;
        def.copies = -1;
        for (int cc : {8, 4, 2, 1}) {
            Shape sh = fit(cc, PAIR_CTAS);
            if (sh.per_sm >= 2) {
                def = sh;
                break;
            }
        }
        if (def.copies < 0) def = fit(1, PAIR_CTAS);
        if (def.per_sm < 1) throw InvalidArg{"pair histogram too large"};
        add(def);
        for (int cc : {8, 4, 2, 1}) add(fit(cc, PAIR_CTAS));
    }
    return out;
}

int grid_for(tpcf_ctx* ctx, const Shape& sh, uint64_t ntasks, int sm_cap) {
    const int sms = sm_cap > 0 ? std::min(sm_cap, ctx->num_sms) : ctx->num_sms;
    uint64_t g = (uint64_t)sms * sh.per_sm;
    if (g > ntasks) g = std::max<uint64_t>(ntasks, 1);
    return (int)g;
}

// Hash of a batch's signature: four chains side by side (26,000 words, those of
// 6,532 voxel jobs: one chain 25 us, four 7; as an array of four, which -O2 keeps
// in memory, 17).
uint64_t batch_key(const std::vector<uint64_t>& sig) {
    const uint64_t m = 1099511628211ull;
    uint64_t a = 1469598103934665603ull, b = 0x9E3779B97F4A7C15ull, c = 0xC2B2AE3D27D4EB4Full, d = 0x165667B19E3779F9ull;
    const uint64_t* w = sig.data();
    const size_t n = sig.size();
    size_t i = 0;
    for (; i + 4 <= n; i += 4) {
        a = (a ^ w[i]) * m;
        b = (b ^ w[i + 1]) * m;
        c = (c ^ w[i + 2]) * m;
        d = (d ^ w[i + 3]) * m;
    }
    for (; i < n; i++) a = (a ^ w[i]) * m;
    uint64_t key = n;
    for (uint64_t x : {a, b, c, d}) key = (key ^ x) * m;
    return key;
}

// Share of the pairs of catalog ranges a and b within `reach`, from 16 points
// spread over a and 256 over b (kept: catalogs do not change); at least half a
// pair of the sample.  Called with ctx->view_mu held.
double pair_share(tpcf_ctx* ctx, const tpcf_job& job, int ra, int rb, const int64_t n[3], float reach) {
    auto key = std::make_tuple(job.catalog[ra], job.begin[ra], n[ra], job.catalog[rb], job.begin[rb], n[rb], reach);
    auto hit = ctx->shares.find(key);
    if (hit != ctx->shares.end()) return hit->second;
    const Catalog &A = *ctx->catalogs.at(job.catalog[ra]), &B = *ctx->catalogs.at(job.catalog[rb]);
    const int64_t sa = std::min<int64_t>(16, n[ra]), sb = std::min<int64_t>(256, n[rb]);
    int within = 0;
    for (int64_t i = 0; i < sa; i++) {
        const int64_t p = job.begin[ra] + i * n[ra] / sa;
        for (int64_t j = 0; j < sb; j++) {
            const int64_t q = job.begin[rb] + j * n[rb] / sb;
            if (p == q && job.catalog[ra] == job.catalog[rb]) continue;
            const float dx = A.x[p] - B.x[q], dy = A.y[p] - B.y[q], dz = A.z[p] - B.z[q];
            within += dx * dx + dy * dy + dz * dz < reach * reach;
        }
    }
    if (ctx->shares.size() >= 65536) ctx->shares.clear();
    return ctx->shares[key] = std::max(0.5, (double)within) / (double)std::max<int64_t>(1, sa * sb);
}

// Whether neighbour lists count a three-side batch sooner than tiles, from the
// shares of its pairs below hist_max.  The coefficients fit the calls' times beyond
// those of any launch, over 950 batches counted both ways (uniform points, clumps
// and sets of small ranges; 60 to 4,000 points, 1 to 1,000 jobs, 1 to 32 bins); the
// rule's choice takes 0.6 % longer than the better of the two on average.
//   Lists: 0.82 ps a pair of a list.  Reference's mode: 4 us and 0.5 ns an
//     accumulator word, for every further job 3 us and 0.4 ns a word, 0.25 us a
//     neighbour of a centre; clean: 1.7 us and 1.15 ns, 7 us and 0.5 ns.
//   Tiles, reference's mode: 0.5 ps a triple (multiset of one catalog), 0.8 ps where
//     a CTA's pipelines share a histogram, and for a multiset accumulator 36 us and
//     1.5 ns a word; clean: 4 ps a triple with two sides in range, 17 ns a tile
//     triple in reach, and a unit's own time, 1.1 us (shared histogram 1.8) a
//     neighbour of its points; for every further job 0.05 ns a word.
// (4,000 points, one catalog, 16 bins to hist_max 180, 90 and 60 in a box of 100:
// lists 8.8, 6.2 and 1.9 ms, tiles 5.3 each; three catalogs 53, 38 and 12, tiles 32.
// Clean, 32 bins: 700 points to 32 lists 99 us, tiles 182; 300 to 12 91 and 78; 300
// jobs of 100 points 4.8 and 0.35 ms.)
bool near_pays(tpcf_ctx* ctx, const Binning& bin, const std::vector<GroupJob>& group, bool shared_hist) {
    const float reach = bin.three.hi;
    const bool clean = bin.three.clean;
    const double words = (double)three_near_acc_words(bin.three.n), more = (double)group.size() - 1;
    double pairs = 0, triples = 0, usable = 0, near_triples = 0, neighbours = 0, multisets = 0;
    std::lock_guard<std::recursive_mutex> vlk(ctx->view_mu);
    const size_t step = (group.size() + 31) / 32;  // (a sample of a large set)
    for (size_t g = 0; g < group.size(); g += step) {
        const tpcf_job& job = *group[g].job;
        int64_t n[3];
        for (int r = 0; r < 3; r++) {
            auto it = ctx->catalogs.find(job.catalog[r]);
            if (it == ctx->catalogs.end()) return true;  // (refused where its view is looked up)
            const int64_t all = it->second->n, end = job.end[r] < 0 ? all : job.end[r];
            if (job.begin[r] < 0 || job.begin[r] > end || end > all) return true;
            n[r] = end - job.begin[r];
        }
        if (n[0] == 0 || n[1] == 0 || n[2] == 0) continue;
        auto same = [&](int a, int b) {
            return job.catalog[a] == job.catalog[b] && job.begin[a] == job.begin[b] && n[a] == n[b];
        };
        // centre and list roles, and the ordered triples of one that is counted
        const bool ab = same(0, 1), bc = same(1, 2), ac = same(0, 2);
        const int c = bc ? 0 : ac ? 1 : ab ? 2 : 0, l1 = c == 0 ? 1 : 0, l2 = c == 2 ? 1 : 2;
        const double by_tiles = ab && bc ? 6 : 1, by_lists = ab && bc ? 6 : ab || bc || ac ? 2 : 1;
        double ordered = (double)n[c], reached = 1;  // triples with two sides in range; share of tile triples in reach
        for (int l : {l1, l2}) {
            const double near = (double)n[l] * pair_share(ctx, job, c, l, n, reach);
            ordered *= near;
            neighbours = std::max(neighbours, near);
            // tiles of 64 points are cbrt(64) mean separations wide
            reached *= std::min(1.0, near / (double)n[l] * pow(1 + cbrt(64 * 4.19 / near), 3));
        }
        const double t = (double)step * (double)n[0] * (double)n[1] * (double)n[2] / by_tiles;
        pairs += (double)step * ordered / by_lists;
        usable += (double)step * ordered / by_tiles;
        triples += t;
        near_triples += reached * t / (TILE * TILE * TILE);
        if (ab && bc) multisets += (double)step;
    }
    double lists = 0.82e-12 * pairs, tiles = 0.05e-9 * words * more;
    if (clean) {
        lists += 1.7e-6 + 1.15e-9 * words + more * (7e-6 + 0.5e-9 * words);
        tiles += 4e-12 * usable + 17e-9 * near_triples + (shared_hist ? 1.8e-6 : 1.1e-6) * std::min(64.0, neighbours);
    } else {
        lists += 4e-6 + 0.5e-9 * words + more * (3e-6 + 0.4e-9 * words) + 0.25e-6 * std::min(150.0, neighbours);
        tiles += (shared_hist ? 0.8e-12 : 0.5e-12) * triples + std::min(3.0, multisets) * (36e-6 + 1.5e-9 * words);
    }
    return lists < tiles;
}

// Runs one group of jobs that share kind, binning and precision in a single
// persistent launch.  outs[i] receives hist_len counts.  lists: counts from
// neighbour lists are allowed; part: the A tiles to count of a single job.
void run_group(tpcf_ctx* ctx, Lane& L, const std::vector<GroupJob>& group, bool lists = true, TileRange part = {}) {
    auto t_wall0 = std::chrono::steady_clock::now();
    const tpcf_spec& sp = *group[0].spec;
    Binning bin = make_binning(sp);
    const int ncat = sp.kind == TPCF_PAIR ? 2 : 3;
    const bool pairs = sp.kind == TPCF_PAIR;
    bool tame = true;  // (asked by the triangle kernels and the neighbour lists only)
    if (!pairs) {
        std::lock_guard<std::recursive_mutex> vlk(ctx->view_mu);
        uint64_t seen[3] = {0, 0, 0};  // (0 is no handle: a role's catalog is often the previous job's)
        for (const GroupJob& g : group)
            for (int r = 0; r < ncat; r++) {
                if (g.job->catalog[r] == seen[r]) continue;
                seen[r] = g.job->catalog[r];
                auto it = ctx->catalogs.find(seen[r]);
                if (it != ctx->catalogs.end()) tame = tame && it->second->tame;
            }
    }
    const bool fp64 = !guarded_fp32(sp, bin, tame);
    bin.tri.tame = tame;
    // three-side counts from neighbour lists (see three_near_kernel)
    const char* near_env = getenv("TPCF_NEAR");
    bool near = lists && bin.near_ok && tame && !(near_env && near_env[0] == '0') &&
                !shape_candidates(ctx, sp, bin, fp64, true, 0).empty() &&
                three_near_acc_words(bin.three.n) * group.size() <= ((size_t)1 << 27);
    if (near && !near_env)
        near = near_pays(ctx, bin, group, shape_candidates(ctx, sp, bin, fp64, false, 0)[0].groups > 0);
    const bool tri_kind = sp.kind == TPCF_TRIANGLE || sp.kind == TPCF_TRIANGLE_JBJ;
    const bool fast_tri = tri_kind && !fp64;
    const bool fast_jbj = sp.kind == TPCF_TRIANGLE_JBJ && !fp64;  // the fast kernel's JBJ binning
    const bool geom = sp.precision == TPCF_GEOMETRY_FP64;
    // Triangles from neighbour lists (see TriCentre) instead of tile triples:
    //   where the tile kernel's tables leave room for one CTA beside the
    //   histogram (50 x 16 x 25 bins, DDD+DDR+DRR+RRR of two seeds: 5k-point cone
    //   4.6 -> 2.0 ms, 5k-point blobs 76 -> 52 ms, 500 points 0.83 -> 0.72 ms;
    //   50 x 16 x 12 bins, two CTAs: blobs 46 -> 51 ms);
    //   where tiles are wide against s_hi (three times), so that few of a tile
    //   triple's triangles are near (1,024 bins: 5k-point cone 0.98 -> 0.68 ms, 2k
    //   0.35 -> 0.19 ms, 500 points 0.14 -> 0.09 ms; blobs, whose tiles are 6 to 20
    //   across, the other way round: 2k 2.2 -> 3.3 ms, 10k 58 -> 64 ms);
    //   JBJ with very many centres, whose tile triples hold few shortest sides
    //   in range (blobs of 25k points, 150,000 centres, 1244 -> 1097 ms, 15k 343 ->
    //   338, 10k 139 -> 140, 5k 24 -> 28 ms; s/m from 0.5: 25k 179 -> 143, 10k 23.4
    //   -> 22.9, 7k 9.9 -> 10.4).  The number of centres stands in for how few of a
    //   tile triple's triangles are near, which depends on the field: of uniform
    //   points the lists are sooner from 5k on (14k in a box of 100 114 -> 74 ms, 5k
    //   9.0 -> 4.6), of many small blobs not at 25k (500 points a blob, 14k 44 ->
    //   57, 25k 164 -> 171).
    // Sets of many small jobs (voxels) keep the tiles: each of a job's centres
    // is an item here (16,500 jobs of a 20k cone 1.9 -> 8.8 ms).
    const char* tl_env = getenv("TPCF_TRI_LISTS");
    bool tlist = lists && fast_tri && bin.list_ok && tame && !(tl_env && tl_env[0] == '0') &&
                 group.size() <= (tl_env ? (size_t)1000000 : (size_t)64) &&
                 !shape_candidates(ctx, sp, bin, fp64, false, 1).empty();
    bool sparse = false;
    if (tlist) {
        uint64_t centres = 0;
        double extent = INFINITY;
        for (const GroupJob& g : group) {
            int64_t n[3];
            for (int r = 0; r < 3; r++) {
                auto v = get_view(ctx, L, g.job->catalog[r], g.job->begin[r], g.job->end[r],
                                  (g.job->flags & TPCF_JOB_GLOBAL_INDEX) != 0);
                n[r] = v->n;
                extent = std::min(extent, v->extent);
            }
            // (a role's points are centres once where roles share a view)
            centres += g.spec->loop == TPCF_LOOP_SAME ? n[0] : n[0] + n[2];
        }
        sparse = extent > 3 * (double)bin.tri.s_hi;
        if (!tl_env)
            tlist = shape_candidates(ctx, sp, bin, fp64, false, 0)[0].per_sm < 2 || sparse ||
                    (fast_jbj && centres >= 80000);
    }
    const bool items = pairs || near || tlist;  // kernels that find their tiles themselves
    if (group.size() > MAX_BATCH_JOBS) throw InvalidArg{"too many jobs in one batch"};
    std::vector<std::pair<const char*, double>> phases;
    auto phase = [&](const char* name) {
        if (plan_trace())
            phases.push_back({name, std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() -
                                                                              t_wall0).count()});
    };
    // device histogram slots: one per job, or one per distinct output for
    // accumulating jobs
    std::vector<size_t> slot_of(group.size());
    std::vector<size_t> slot_job;  // first job of each slot
    {
        std::unordered_map<uint64_t*, size_t> by_out;
        for (size_t g = 0; g < group.size(); g++) {
            if (group[g].accumulate) {
                auto ins = by_out.emplace(group[g].out, slot_job.size());
                slot_of[g] = ins.first->second;
                if (!ins.second) continue;
            }
            slot_of[g] = slot_job.size();
            slot_job.push_back(g);
        }
    }
    const size_t nslots = slot_job.size();
    size_t hist_total = (size_t)bin.len * nslots;
    L.d_hist.reserve(hist_total);
    const char* rdd_env = getenv("TPCF_RDD");
    const bool rdd = fast_tri && !(rdd_env && rdd_env[0] == '0');
    const char* sym_env = getenv("TPCF_SYM3");
    const bool sym_three = !(sym_env && sym_env[0] == '0');
    // The distinct catalog ranges of the batch (a batch of many jobs names
    // few): each is looked up once, and its view -- which may still be being
    // built (new catalogs) -- is waited for only when the batch is planned.
    struct RangeKey {
        uint64_t h;
        int64_t b, e;
        bool gl;
        bool operator==(const RangeKey& o) const { return h == o.h && b == o.b && e == o.e && gl == o.gl; }
    };
    struct RangeHash {
        size_t operator()(const RangeKey& k) const {
            uint64_t x = k.h * 0x9E3779B97F4A7C15ull ^ (uint64_t)k.b * 0xC2B2AE3D27D4EB4Full ^
                         (uint64_t)k.e * 0x165667B19E3779F9ull ^ (uint64_t)k.gl;
            return (size_t)(x ^ (x >> 29));
        }
    };
    struct Range {
        RangeKey key;
        ViewRef ref;
        std::shared_ptr<View> view;
    };
    std::vector<Range> ranges;
    std::unordered_map<RangeKey, uint32_t, RangeHash> range_at;
    // the last range of each hash value: a batch of thousands of jobs names
    // each of its ranges many times
    size_t nfront = 1;
    while (nfront < 3 * group.size() && nfront < 4096) nfront *= 2;
    std::vector<uint32_t> front(nfront, UINT32_MAX);
    auto range_of = [&](const RangeKey& k) -> uint32_t {
        uint32_t& f = front[RangeHash{}(k) & (nfront - 1)];
        if (f != UINT32_MAX && ranges[f].key == k) return f;
        auto ins = range_at.try_emplace(k, (uint32_t)ranges.size());
        if (ins.second) {
            Range r{k, {}, nullptr};
            get_view(ctx, L, k.h, k.b, k.e, k.gl, &r.ref);
            ranges.push_back(std::move(r));
        }
        return f = ins.first->second;
    };
    // Signature of the batch (its binning, and each job's views, slot and loop
    // nest): a repeated batch over the same resident views reuses its plan.
    std::vector<uint64_t> sig;
    sig.reserve(17 + group.size() * 4);
    sig.push_back((uint64_t)(uintptr_t)L.d_hist.p);
    {
        const uint64_t f[6] = {(uint64_t)sp.kind, (uint64_t)sp.prune, (uint64_t)sp.precision, (uint64_t)sp.nan_policy,
                               (uint64_t)sp.overflow, (uint64_t)tlist << 3 | (uint64_t)near << 2 | (uint64_t)rdd << 1 | (uint64_t)sym_three};
        sig.insert(sig.end(), f, f + 6);
        for (int a = 0; a < 3; a++) {
            sig.push_back((uint64_t)fbits(sp.axis[a].lo) << 32 | fbits(sp.axis[a].hi));
            sig.push_back((uint64_t)(uint32_t)sp.axis[a].nbins);
        }
        sig.push_back((uint64_t)bin.len);
        sig.push_back((uint64_t)group.size());
        sig.push_back((uint64_t)(uint32_t)part.begin << 32 | (uint32_t)part.end);
    }
    // each job: its ranges in the kernel's role order, and how its tiles and
    // points are enumerated (JOB_*)
    struct RoleJob {
        uint32_t range[3];
        uint32_t mode;
    };
    std::vector<RoleJob> roles(group.size());
    // triangles from neighbour lists: what is launched instead of the jobs
    struct SubJob {
        uint32_t range[3], mode, job;
    };
    std::vector<SubJob> subs;
    uint64_t units = 0;
    // reference loop size of job g
    auto job_units = [&](size_t g) {
        const tpcf_job& job = *group[g].job;
        int64_t n[3] = {0, 0, 0};
        for (int r = 0; r < ncat; r++)
            n[r] = ranges[range_of({job.catalog[r], job.begin[r], job.end[r],
                                    (job.flags & TPCF_JOB_GLOBAL_INDEX) != 0})].ref.n;
        return loop_units(group[g].spec->kind, group[g].spec->loop, n);
    };
    // a role's range is often the previous job's
    RangeKey last_key[3] = {};
    uint32_t last_at[3] = {};
    bool last_ok[3] = {};
    for (size_t g = 0; g < group.size(); g++) {
        const tpcf_job& job = *group[g].job;
        const tpcf_spec& jsp = *group[g].spec;  // same binning as sp; the loop nest may differ
        int64_t n[3] = {0, 0, 0};
        uint32_t rg[3] = {0, 0, 0};
        for (int r = 0; r < ncat; r++) {
            const RangeKey k{job.catalog[r], job.begin[r], job.end[r], (job.flags & TPCF_JOB_GLOBAL_INDEX) != 0};
            if (!last_ok[r] || !(last_key[r] == k)) {
                last_at[r] = range_of(k);
                last_key[r] = k;
                last_ok[r] = true;
            }
            rg[r] = last_at[r];
            n[r] = ranges[rg[r]].ref.n;
        }
        if (ncat == 2) rg[2] = rg[1];
        if (part.begin == 0) units += loop_units(jsp.kind, jsp.loop, n);  // (a job's first part reports it)
        // (two ranges with one view, e.g. [0, n) and [0, -1), are the same array)
        auto id = [&](int r) { return ranges[rg[r]].ref.id; };
        const bool ab = id(0) == id(1), bc = id(1) == id(2);
        uint32_t mode = PRED_NONE, v[3] = {rg[0], rg[1], rg[2]};
        if (tlist) {
            // the job's triangles by the role of their centre: each with its
            // lists' views (one view: its unordered pairs)
            uint32_t pred = PRED_NONE;
            uint32_t rank[3] = {0, 1, 2};
            auto sub = [&](int rc, int r1, int r2, bool self) {
                SubJob sj{};
                sj.range[0] = rg[rc], sj.range[1] = rg[r1], sj.range[2] = rg[r2];
                sj.job = (uint32_t)g;
                sj.mode = pred | (self ? TL_SELF : 0u) | (uint32_t)(rc | r1 << 2 | r2 << 4) << TL_ROLE_SHIFT |
                          (rank[rc] | rank[r1] << 2 | rank[r2] << 4) << TL_RANK_SHIFT;
                subs.push_back(sj);
            };
            if (ab && bc && jsp.loop == TPCF_LOOP_SAME) {
                rank[1] = rank[2] = 0;
                sub(0, 1, 2, true);
            } else if (ab && !bc && jsp.loop == TPCF_LOOP_ONE) {
                pred = PRED_DDR;
                rank[1] = 0;
                sub(2, 0, 1, true);
                sub(0, 1, 2, false);
            } else if (bc && !ab && jsp.loop == TPCF_LOOP_ONE) {
                rank[2] = rank[1];
                sub(0, 1, 2, true);
                sub(1, 0, 2, false);
            } else {
                pred = jsp.loop == TPCF_LOOP_SAME ? PRED_SAME : jsp.loop == TPCF_LOOP_ONE ? PRED_ONE : PRED_NONE;
                sub(0, 1, 2, false);
                sub(1, 0, 2, false);
                sub(2, 0, 1, false);
            }
        } else if (near) {
            // the centre: the point of the view that appears once, or any
            const bool ac = id(0) == id(2);
            if (ab && bc && sym_three) {
                mode = NEAR_SYM;
            } else if (bc) {
                mode = NEAR_PAIR;
            } else if (ac) {
                v[0] = rg[1], v[1] = v[2] = rg[0];
                mode = NEAR_PAIR | 1u << NEAR_CENTRE_SHIFT;
            } else if (ab) {
                v[0] = rg[2], v[1] = v[2] = rg[0];
                mode = NEAR_PAIR | 2u << NEAR_CENTRE_SHIFT;
            } else {
                mode = NEAR_ORDERED;
            }
        } else if (pairs) {
            if (jsp.loop == TPCF_LOOP_SAME) mode = ab ? JOB_B_FROM_A : (uint32_t)PRED_SAME;
        } else if (tri_kind && jsp.loop == TPCF_LOOP_ONE && ab && !bc && rdd) {
            // Loop ONE jobs of two arrays are counted with the point of the
            // array that appears once in role B or C and the pair array
            // first, so that points out of reach of a tile are skipped whole:
            // D-D-R (A == B) in the roles (C, A, A), each point of C with
            // every unordered pair of the single array ...
            v[0] = rg[2], v[1] = v[2] = rg[0];
            mode = PRED_RDD | JOB_C_FROM_B;
        } else if (tri_kind && jsp.loop == TPCF_LOOP_ONE && bc && !ab && rdd) {
            // ... and D-R-R (B == C) in the roles (B, B, A), every unordered
            // pair of the pair array with each point of the other
            v[0] = v[1] = rg[1], v[2] = rg[0];
            mode = PRED_NONE | JOB_B_FROM_A;
        } else if (ab && bc && tri_kind && jsp.loop == TPCF_LOOP_SAME) {
            // i <= j <= k over one array: unordered distinct triples
            mode = PRED_NONE | JOB_B_FROM_A | JOB_C_FROM_B;
        } else if (ab && bc && sp.kind == TPCF_THREE_SIDE && jsp.loop == TPCF_LOOP_ALL && sym_three) {
            // three-side histogram of one catalog in all roles: the kernel
            // counts each multiset {i, j, k} once for all its orderings
            mode = PRED_SAME | JOB_B_FROM_A | JOB_C_FROM_B;
        } else if (tri_kind && jsp.loop == TPCF_LOOP_ONE && bc) {
            // j <= k over one array (j == k has a zero side): unordered pairs
            mode = PRED_NONE | JOB_C_FROM_B;
        } else if (tri_kind && jsp.loop == TPCF_LOOP_ONE && ab) {
            // every ordered (i, j) of one array, k >= j: unordered {i, j} with
            // weight [k >= i] + [k >= j]
            mode = PRED_DDR | JOB_B_FROM_A;
        } else if (tri_kind) {
            mode = jsp.loop == TPCF_LOOP_SAME ? PRED_SAME : jsp.loop == TPCF_LOOP_ONE ? PRED_ONE : PRED_NONE;
        }
        roles[g] = {{v[0], v[1], v[2]}, mode};
        sig.push_back(ranges[v[0]].ref.id);
        sig.push_back(ranges[v[1]].ref.id);
        sig.push_back(ranges[v[2]].ref.id);
        sig.push_back((uint64_t)slot_of[g] << 32 | (uint64_t)mode << 8 | (uint64_t)jsp.loop);
    }
    // neighbour lists: an accumulator per output slot and class of job, and the
    // wedge jobs of the reference's mode (two per job, one for a single catalog)
    std::vector<uint32_t> acc_of;
    std::vector<std::pair<size_t, uint32_t>> accs;  // slot, mode
    const size_t acc_words = near ? three_near_acc_words(bin.three.n) : 0;
    size_t nwedge_jobs = 0;
    if (near) {
        std::map<std::pair<size_t, uint32_t>, uint32_t> at;
        for (size_t g = 0; g < group.size(); g++) {
            auto ins = at.emplace(std::make_pair(slot_of[g], roles[g].mode), (uint32_t)accs.size());
            if (ins.second) accs.push_back(ins.first->first);
            acc_of.push_back(ins.first->second);
            if (!bin.three.clean) nwedge_jobs += roles[g].mode == NEAR_SYM ? 1 : 2;
        }
        // (the planned jobs point into it, as into the histograms)
        L.d_acc.reserve(acc_words * accs.size());
        sig.push_back((uint64_t)(uintptr_t)L.d_acc.p);
    }
    cudaStream_t st = L.stream;
    L.d_counters.reserve(CTR_WORDS);
    const std::vector<Shape> cands = shape_candidates(ctx, sp, bin, fp64, near, tlist ? (int)nslots : 0);
    const bool plan_hit = sig == L.plan_sig;
    // of the batch, in what is remembered of it (without lists it is asked for only
    // when the plan is under way on the device)
    uint64_t key = 0;
    if (near) {
        key = batch_key(sig);
        bool refused = false;
        {
            std::lock_guard<std::mutex> tlk(ctx->tune_mu);
            refused = ctx->refused.count(key) > 0;
        }
        if (refused) return run_group(ctx, L, group, false);
    }
    phase("batch");
    // (plain FP64 one A tile at a time, so that CTAs side by side take unlike tiles B
    // and C: three-side DDD+DRR of 400 points 0.65 -> 0.55 ms)
    const int window = fp64                   ? 1
                       : ctx->group_tasks > 0 ? std::min(ctx->group_tasks, MAX_WINDOW)
                                              : (group.size() > 64 ? 16 : 4);
    uint32_t nrows = L.plan_rows;   // pairs and neighbour lists: items
    int plan_chunk = L.plan_chunk;  // pairs: tiles B per item; neighbour lists: centres per item
    uint32_t nwedges = L.plan_wedges;
    int plan_parts = L.plan_parts, plan_kparts = L.plan_kparts;  // triangle lists: shares of a centre
    PlanHeader* d_header = nullptr;
    const uint32_t unit_limit = plan_limit("TPCF_MAX_UNITS", MAX_UNITS),
                   row_limit = plan_limit("TPCF_MAX_ROWS", items ? MAX_ITEMS : MAX_ROWS);
    auto too_large = [&] {
        const int tile = ctx->tile_points;
        L.plan_sig.clear();
        return TooLarge{part.end < 0 ? (int)((ranges[roles[0].range[0]].ref.n + tile - 1) / tile) : part.end - part.begin,
                        near || tlist};
    };
    // Finds the units of the batch on the device (see plan_rows): the host
    // gives each job's number of rows.
    auto plan_units = [&](size_t capacity) {
        L.d_units.reserve(capacity);
        L.d_masks.reserve(capacity);
        PlanParams pp{};
        pp.window = window;
        pp.per_tile = fast_tri ? 0 : 1;
        // (A part makes the unit's j-k table again.  That is most of the work where
        // sides are computed in FP64, or where clean mode leaves few triples:
        // three-side DDD+DRR of 400 points in plain FP64 0.57 ms whole, 0.83 cut; a
        // clean D-D-R of 1,000 points, hist_max a tenth of the box, 31 and 42 us.)
        pp.max_parts = fast_tri ? 16 : sp.kind == TPCF_THREE_SIDE && (fp64 || bin.three.clean) ? 1 : 4;
        pp.tri = bin.tri_prune ? 1 : 0;
        pp.slots = grid_for(ctx, cands[0], UINT64_MAX, L.sm_cap) * std::max(1, cands[0].groups);
        const double l2 = bin.lmax * bin.lmax;
        pp.lmax2 = l2 < 3e38 ? nextafterf((float)l2, INFINITY) : INFINITY;
        auto sq_up = [](double v) { return v > 0 ? (v * v < 3e38 ? nextafterf((float)(v * v), INFINITY) : INFINITY) : 0.f; };
        pp.s_hi2 = sq_up(bin.s_hi);
        pp.q_hi2 = sq_up(bin.q_hi);
        pp.s_lo2 = bin.s_lo > 0 ? nextafterf((float)std::min(bin.s_lo * bin.s_lo, 3e38), 0.f) : 0.f;
        // heavy: what takes a CTA that has its SM to itself some 12 us (a line
        // at 6000 or 8192 instead cost 1 % on 10k points and 2 % on 1k; at 1500
        // 1k points are 4 % faster and a burst of 40 mixed jobs 8 % slower)
        pp.r = (float)(bin.lmax < 3e38 ? (sp.kind == TPCF_TRIANGLE ? std::max(0.0, bin.s_hi * bin.q_hi) : bin.lmax) : 3e38);
        pp.heavy = fast_tri ? 3000.f : 0.f;
        int rpb = 0;
        const int blocks = plan_blocks(nrows, &rpb);
        L.d_row_cnt.reserve(std::max<size_t>(nrows, 1));
        L.d_block_sum.reserve((size_t)blocks + 1);
        CK(launch_plan(L.d_jobs.p, L.d_rows.p, (int)group.size(), nrows, pp, L.d_row_cnt.p, L.d_block_sum.p, d_header,
                       L.d_units.p, L.d_masks.p, (uint32_t)capacity, st));
    };
    d_header = reinterpret_cast<PlanHeader*>(L.d_counters.p + CTR_HEADER);
    if (!plan_hit) {
        L.plan_sig.clear();  // (set again once the plan is on the device)
        for (Range& r : ranges) r.view = get_view(ctx, L, r.key.h, r.key.b, r.key.e, r.key.gl);
        phase("views");
        CK(cudaStreamSynchronize(st));  // (a failed batch may still read the pinned buffers)
        const size_t njobs = tlist ? subs.size() : group.size() + nwedge_jobs + accs.size();
        L.h_jobs.reserve(njobs);
        L.h_rows.reserve(njobs + 2);
        uint64_t rows = 0;
        plan_chunk = 0;
        if (pairs) {
            long long tile_pairs = 0;
            for (const RoleJob& r : roles)
                tile_pairs += (long long)ranges[r.range[0]].view->ntiles * ranges[r.range[1]].view->ntiles;
            plan_chunk = pair_chunk(tile_pairs, ctx->num_sms * PAIR_CTAS, fp64);
        } else if (near) {
            // one centre per item where that balances the pipelines, else as
            // many as an item may have
            uint64_t centres = 0;
            bool ordered = false;
            for (const RoleJob& r : roles) {
                centres += ranges[r.range[0]].view->n;
                ordered = ordered || r.mode == NEAR_ORDERED;
            }
            plan_chunk = centres < 64ull * ctx->num_sms * 4 ? 1 : ordered ? NEAR_ITEM_ORDERED : NEAR_ITEM;
        } else if (tlist) {
            uint64_t centres = 0;
            for (const SubJob& sj : subs) centres += ranges[sj.range[0]].view->n;
            const uint64_t warps = (uint64_t)ctx->num_sms * TL_MAX_WARPS;
            plan_chunk = centres < 64 * warps ? 1 : 4;
            plan_parts = 1;
            plan_kparts = 1;
            // (J's shares first: a share of K's fills its J lists again; a sparse
            // view's centres are light)
            while (plan_parts * plan_kparts < (sparse ? 2 : 64) && centres * plan_parts * plan_kparts < TL_WANT * warps)
                if (plan_parts < 16) plan_parts *= 2;
                else plan_kparts *= 2;
            for (size_t k = 0; k < subs.size(); k++) {
                DevJob d{};
                for (int r = 0; r < 3; r++) {
                    const View& v = *ranges[subs[k].range[r]].view;
                    d.pts[r] = v.pts.p;
                    d.tile_start[r] = v.tile_start.p;
                    d.box[r] = v.box.p;
                    d.ntiles[r] = v.ntiles;
                }
                d.mode = subs[k].mode;
                d.hist = L.d_hist.p + (size_t)bin.len * slot_of[subs[k].job];
                d.weight = (unsigned long long)ranges[subs[k].range[0]].view->n | (unsigned long long)slot_of[subs[k].job] << 32;
                L.h_jobs.p[k] = d;
                L.h_rows.p[k] = (uint32_t)rows;
                rows += (uint64_t)plan_parts * plan_kparts * (((uint64_t)ranges[subs[k].range[0]].view->n + plan_chunk - 1) / plan_chunk);
                if (rows > row_limit) throw too_large();
            }
        }
        for (size_t g = 0; g < (tlist ? 0 : group.size()); g++) {
            DevJob d{};
            for (int r = 0; r < 3; r++) {
                const View& v = *ranges[roles[g].range[r]].view;
                d.pts[r] = v.pts.p;
                d.tile_start[r] = v.tile_start.p;
                d.box[r] = v.box.p;
                d.ntiles[r] = v.ntiles;
            }
            d.mode = roles[g].mode;
            d.hist = L.d_hist.p + (size_t)bin.len * slot_of[g];
            if (part.end >= 0) {
                // tables that begin with the first A tile; tiles B >= A then begin
                // there as well, and tiles C >= B with them
                d.ntiles[0] = part.end;
                for (int r = 0; r < 3; r++) {
                    if (r == 1 && !(d.mode & JOB_B_FROM_A)) break;
                    if (r == 2 && !(d.mode & JOB_C_FROM_B)) break;
                    d.tile_start[r] += part.begin;
                    d.box[r] += 2 * (size_t)part.begin;
                    d.ntiles[r] -= part.begin;
                }
            }
            L.h_jobs.p[g] = d;
            L.h_rows.p[g] = (uint32_t)rows;
            if (near) {
                L.h_jobs.p[g].hist = L.d_acc.p + acc_words * acc_of[g];
                rows += (uint64_t)d.ntiles[0] * ((TILE + plan_chunk - 1) / plan_chunk);
            } else if (pairs) rows += (uint64_t)d.ntiles[0] * ((d.ntiles[1] + plan_chunk - 1) / plan_chunk);
            else if (d.ntiles[2] > 0) rows += (uint64_t)((d.ntiles[0] + window - 1) / window) * d.ntiles[1];
            if (rows > row_limit) throw too_large();
        }
        size_t nr = tlist ? subs.size() : group.size();
        L.h_rows.p[nr++] = (uint32_t)rows;
        nrows = (uint32_t)rows;
        if (near) {
            // wedge jobs: pairs of sides at a point of role B (lists A, C; the
            // pairs B-C weigh the points of A) and of role C (lists A, B)
            const size_t m = bin.three.n + 1;
            uint64_t w = 0;
            size_t at = group.size();
            for (size_t g = 0; nwedge_jobs && g < group.size(); g++) {
                const uint32_t centre = roles[g].mode >> NEAR_CENTRE_SHIFT;
                // the views of the reference's roles
                const int of[3][3] = {{0, 1, 2}, {1, 0, 2}, {1, 2, 0}};
                const View* v[3];
                for (int r = 0; r < 3; r++) v[r] = ranges[roles[g].range[of[centre][r]]].view.get();
                const bool sym = roles[g].mode == NEAR_SYM;
                unsigned long long* acc = L.d_acc.p + acc_words * acc_of[g] + m * m * m + m + 1;
                for (int k = 0; k < (sym ? 1 : 2); k++) {
                    const View* role[3] = {v[1 + k], v[0], v[2 - k]};
                    DevJob d{};
                    for (int r = 0; r < 3; r++) {
                        d.pts[r] = role[r]->pts.p;
                        d.tile_start[r] = role[r]->tile_start.p;
                        d.box[r] = role[r]->box.p;
                        d.ntiles[r] = role[r]->ntiles;
                    }
                    d.mode = sym ? NEAR_SYM : NEAR_ORDERED;
                    d.hist = acc + k * m * m;
                    d.aux = k == 0 ? acc + 2 * m * m : nullptr;
                    d.weight = (unsigned long long)v[0]->n;
                    L.h_jobs.p[at] = d;
                    L.h_rows.p[nr++] = (uint32_t)w;
                    w += (uint64_t)d.ntiles[0] * 8;
                    if (w > row_limit) throw too_large();
                    at++;
                }
            }
            L.h_rows.p[nr++] = (uint32_t)w;
            nwedges = (uint32_t)w;
            for (const auto& a : accs) {
                DevJob d{};
                d.mode = a.second;
                d.hist = L.d_acc.p + acc_words * (size_t)(&a - accs.data());
                d.aux = L.d_hist.p + (size_t)bin.len * a.first;
                L.h_jobs.p[at++] = d;
            }
        }
        L.d_jobs.reserve(njobs);
        L.d_rows.reserve(nr);
        CK(cudaMemcpyAsync(L.d_jobs.p, L.h_jobs.p, njobs * sizeof(DevJob), cudaMemcpyHostToDevice, st));
        CK(cudaMemcpyAsync(L.d_rows.p, L.h_rows.p, nr * sizeof(uint32_t), cudaMemcpyHostToDevice, st));
        L.h2d += njobs * sizeof(DevJob) + nr * sizeof(uint32_t);
        if (!items) plan_units(std::min<size_t>(std::max<size_t>(L.d_units.n, (size_t)1 << 20), unit_limit));
        L.plan_sig = sig;
        L.plan_rows = nrows;
        L.plan_chunk = plan_chunk;
        L.plan_wedges = nwedges;
        L.plan_parts = plan_parts;
        L.plan_kparts = plan_kparts;
        phase("plan");
    }
    L.stats.plan_ms =
        std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t_wall0).count();
    if (sp.kind == TPCF_TRIANGLE) ensure_acos(ctx);
    const AcosTable acos_t = sp.kind == TPCF_TRIANGLE ? acos_table(ctx) : AcosTable{};
    // guard-band triangles are queued and recomputed (JBJ tiles: in the kernel)
    const bool recheck = fast_tri && (!fast_jbj || tlist);
    uint64_t launches = recheck ? 2 : 1;  // counting (+ recheck)
    const char* genv = getenv("TPCF_GRAPHS");
    const bool graphs = L.graphs_ok && !(genv && genv[0] == '0');
    L.h_hist.reserve(hist_total);
    L.h_counters.reserve(CTR_WORDS);
    // recheck queue: at least 4M entries; TPCF_RECHECK_CAP lowers the floor
    // (tests use it to run the overflow path: grow the queue, count again)
    size_t queue_floor = (size_t)1 << 22;
    if (const char* qc = getenv("TPCF_RECHECK_CAP")) queue_floor = (size_t)std::max(1L, std::atol(qc));
    unsigned int queue_cap = (unsigned int)std::max<size_t>(L.d_queue.n, queue_floor);
    uint64_t dev_evaluated = 0, dev_binned = 0, replays = 0, regrows = 0;
    PlanHeader header{};
    // units (pairs: items) known on the host: needed where a batch is counted in slices
    bool sized = items;
    uint32_t nwork = items ? nrows : 0xffffffffu;

    // One complete count of the group with launch shape sh: zero, count,
    // recheck, copy back (replayed from a captured graph when allowed and
    // the batch repeats).  Returns the device time in ms.
    auto count_with = [&](const Shape& sh, bool allow_graph) -> float {
        const int copies = sh.copies;
        const int grid = grid_for(ctx, sh, items ? (nrows + std::max(1, sh.groups) - 1) / std::max(1, sh.groups) : UINT64_MAX, L.sm_cap);
        for (int attempt = 0;; attempt++) {
            // (the unit list and the recheck queue grow at most once each)
            if (attempt == 4) throw InternalError{"a batch overflowed its buffers after they had been grown"};
            if (L.slice_batches && !sized) {
                // (the header of a plan that overflowed the unit list asks for a
                // larger one: the count below finds no units and regrows it)
                CK(cudaMemcpyAsync(L.h_counters.p, L.d_counters.p, CTR_WORDS * sizeof(unsigned int),
                                   cudaMemcpyDeviceToHost, st));
                CK(cudaStreamSynchronize(st));
                memcpy(&header, L.h_counters.p + CTR_HEADER, sizeof(header));
                nwork = header.nunits;
                sized = true;
            }
            // slices of at least 8 units per CTA, at most 64 of them
            unsigned int slice = L.slice_batches ? std::max<unsigned int>((unsigned int)grid * 8u, (nwork + 63u) / 64u)
                                                 : std::max(nwork, 1u);
            if (L.slice_batches && ctx->slice_tasks > 0) slice = (unsigned int)ctx->slice_tasks;
            launches = (nwork > slice ? (nwork + slice - 1) / slice : 1) +
                       (recheck ? 1 : near ? (nwedges ? 2 : 1) : 0);
            RecheckQueue q{};
            q.hists = L.d_hist.p;
            if (recheck) {
                if (L.d_queue.n < queue_cap) L.drop_graph();
                L.d_queue.reserve(queue_cap);
                q.items = L.d_queue.p;
                q.count = L.d_counters.p + CTR_RECHECK;
                q.cap = queue_cap;
                q.evaluated = reinterpret_cast<unsigned long long*>(L.d_counters.p + CTR_EVAL);
            } else if (fast_jbj) {
                q.count = L.d_counters.p + CTR_RECHECK;  // no item is ever queued (cap 0)
                q.evaluated = reinterpret_cast<unsigned long long*>(L.d_counters.p + CTR_EVAL);
            }
            auto enqueue = [&](bool capturing) -> cudaError_t {
                const unsigned int ev_flags = capturing ? cudaEventRecordExternal : cudaEventRecordDefault;
                cudaError_t e;
#define EQ(x)                                   \
    do {                                        \
        if ((e = (x)) != cudaSuccess) return e; \
    } while (0)
                EQ(cudaMemsetAsync(L.d_hist.p, 0, hist_total * sizeof(unsigned long long), st));
                EQ(cudaMemsetAsync(L.d_counters.p, 0, CTR_ZEROED * sizeof(unsigned int), st));
                if (near) EQ(cudaMemsetAsync(L.d_acc.p, 0, acc_words * accs.size() * sizeof(unsigned long long), st));
                EQ(cudaEventRecordWithFlags(L.ev0, st, ev_flags));
                // the counting kernel over units (items) [t0, t0 + n)
                auto launch_main = [&](unsigned int t0, unsigned int n) -> cudaError_t {
                    unsigned int* counter = L.d_counters.p + CTR_WORK;
                    const UnitList ul{d_header, L.d_units.p, L.d_masks.p, t0, n};
                    if (tlist)
                        return launch_tri_list(L.d_jobs.p, L.d_rows.p, (int)subs.size(), t0, n, plan_chunk, plan_parts,
                                               plan_kparts, copies,
                                               counter, bin.tri, q, grid, sh.groups, fast_jbj ? 1 : geom ? 2 : 0, st);
                    if (fast_tri)  // (JBJ: exact without a recheck)
                        return launch_triangle_fast(L.d_jobs.p, ul, counter, bin.tri, q, grid, copies,
                                                    fast_jbj ? 1 : geom ? 2 : 0, st);
                    if (tri_kind)
                        return launch_triangle_fp64(L.d_jobs.p, ul, counter, bin.tri, acos_t, grid, copies,
                                                    sp.kind == TPCF_TRIANGLE_JBJ ? 2
                                                    : geom ? 1 : 0, st);
                    if (near)
                        return launch_three_near(L.d_jobs.p, L.d_rows.p, (int)group.size(), t0, n, plan_chunk, counter,
                                                 L.d_counters.p + CTR_DENSE,
                                                 reinterpret_cast<unsigned long long*>(L.d_counters.p + CTR_EVAL),
                                                 bin.near, grid, sh.groups, st);
                    if (sp.kind == TPCF_THREE_SIDE)
                        return launch_three_side(L.d_jobs.p, ul, counter, bin.three, fp64, grid, copies, sh.groups, st);
                    return launch_pairs(L.d_jobs.p, L.d_rows.p, (int)group.size(), t0, n, plan_chunk, counter,
                                        reinterpret_cast<unsigned long long*>(L.d_counters.p + CTR_EVAL), bin.pair, fp64,
                                        grid, copies, st);
                };
                // one launch over all units, or (a heavy serving batch) slices of
                // them, between which the device can start the kernels that
                // higher-priority streams (the light serving lanes) have queued
                EQ(launch_main(0, std::min(nwork, slice)));
                for (unsigned int t0 = slice; t0 < nwork; t0 += slice) {
                    EQ(cudaMemsetAsync(L.d_counters.p + CTR_WORK, 0, sizeof(unsigned int), st));  // the slice's counter
                    EQ(launch_main(t0, std::min(slice, nwork - t0)));
                }
                EQ(cudaEventRecordWithFlags(L.ev_mid, st, ev_flags));
                if (near) {
                    const DevJob* after = L.d_jobs.p + group.size();
                    EQ(launch_three_wedges(after, L.d_rows.p + group.size() + 1, (int)nwedge_jobs, nwedges,
                                           L.d_counters.p + CTR_DENSE, bin.near, ctx->num_sms * 8, st));
                    EQ(launch_three_expand(after + nwedge_jobs, (int)accs.size(), bin.near, st));
                }
                if (recheck)
                    EQ(launch_triangle_recheck(L.d_jobs.p, q, bin.tri, acos_t, fast_jbj ? 1 : geom ? 2 : 0,
                                               ctx->num_sms * 8, st));
                EQ(cudaEventRecordWithFlags(L.ev1, st, ev_flags));
                EQ(cudaMemcpyAsync(L.h_counters.p, L.d_counters.p, CTR_WORDS * sizeof(unsigned int),
                                   cudaMemcpyDeviceToHost, st));
                EQ(cudaMemcpyAsync(L.h_hist.p, L.d_hist.p, hist_total * sizeof(unsigned long long),
                                   cudaMemcpyDeviceToHost, st));
#undef EQ
                return cudaSuccess;
            };
            bool replayed = false;
            if (allow_graph) {
                // everything the captured launches read: the batch, its buffers, the shape
                std::vector<uint64_t> gsig = sig;
                const uint64_t extra[] = {(uint64_t)(uintptr_t)L.d_jobs.p, (uint64_t)(uintptr_t)L.d_units.p,
                                          (uint64_t)(uintptr_t)L.d_counters.p, (uint64_t)(uintptr_t)L.d_queue.p,
                                          (uint64_t)(uintptr_t)L.h_hist.p, (uint64_t)(uintptr_t)L.h_counters.p,
                                          (uint64_t)(uintptr_t)acos_t.keys, (uint64_t)(uintptr_t)acos_t.vals,
                                          (uint64_t)(uintptr_t)acos_t.bucket, (uint64_t)acos_t.n, queue_cap,
                                          (uint64_t)grid, (uint64_t)copies, (uint64_t)sh.groups, hist_total,
                                          (uint64_t)nwork, (uint64_t)slice, (uint64_t)(uintptr_t)L.d_rows.p,
                                          (uint64_t)(uintptr_t)L.d_masks.p, (uint64_t)plan_chunk, (uint64_t)plan_parts << 32 | (uint64_t)plan_kparts};
                gsig.insert(gsig.end(), extra, extra + sizeof(extra) / sizeof(extra[0]));
                if (!L.graph || gsig != L.graph_sig) {
                    L.drop_graph();
                    cudaGraph_t g = nullptr;
                    cudaError_t e = cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal);
                    if (e == cudaSuccess) {
                        cudaError_t e1 = enqueue(true);
                        cudaError_t e2 = cudaStreamEndCapture(st, &g);
                        e = e1 != cudaSuccess ? e1 : e2;
                    }
                    if (e == cudaSuccess) e = cudaGraphInstantiate(&L.graph, g, 0);
                    if (g) cudaGraphDestroy(g);
                    if (e == cudaSuccess) {
                        L.graph_sig = gsig;
                    } else {
                        // capture unavailable here: issue the launches one by one from now on
                        (void)cudaGetLastError();
                        L.graph = nullptr;
                        L.graphs_ok = false;
                    }
                }
                if (L.graph) {
                    CK(cudaGraphLaunch(L.graph, st));
                    replayed = true;
                }
            }
            if (!replayed) CK(enqueue(false));
            CK(cudaStreamSynchronize(st));
            replays = replayed ? 1 : 0;
            const unsigned int* counters = L.h_counters.p;
            L.d2h += CTR_WORDS * sizeof(unsigned int) + hist_total * sizeof(unsigned long long);
            memcpy(&header, counters + CTR_HEADER, sizeof(header));
            if (!items && header.mismatch) {
                L.plan_sig.clear();
                throw InternalError{"the planner's passes found different units"};
            }
            if (!items && header.nunits == 0 && header.needed > 0) {
                // the unit list overflowed: nothing was counted; plan again into a larger one
                L.drop_graph();
                if (header.needed > unit_limit) throw too_large();
                plan_units(std::min<size_t>((size_t)header.needed + (header.needed >> 3), unit_limit));
                sized = false;
                continue;
            }
            L.stats.recheck_units = counters[CTR_RECHECK];
            memcpy(&dev_evaluated, &counters[CTR_EVAL], sizeof(dev_evaluated));
            memcpy(&dev_binned, &counters[CTR_EVAL + 2], sizeof(dev_binned));
            if (recheck && counters[CTR_RECHECK] > queue_cap) {
                // the recheck queue overflowed: grow it and count again
                queue_cap = (unsigned int)std::min<uint64_t>(
                    (uint64_t)counters[CTR_RECHECK] + (counters[CTR_RECHECK] >> 2) + 1024, 0xF0000000ull);
                regrows++;
                continue;
            }
            break;
        }
        float t = 0;
        CK(cudaEventElapsedTime(&t, L.ev0, L.ev1));
        return t;
    };

    // Launch shape: the tuned one for this batch if the autotuner has seen it,
    // else the default.  A batch that repeats (its plan was cached) and has no
    // tuned shape yet is counted once with every candidate shape -- each count
    // is exact -- and the fastest is kept for the next calls.
    const char* tenv = getenv("TPCF_AUTOTUNE");
    const bool autotune = !(tenv && tenv[0] == '0');
    Shape shape = cands[0];
    uint64_t tuned_runs = 0;
    if (!near) key = batch_key(sig);
    {
        std::lock_guard<std::mutex> tlk(ctx->tune_mu);
        auto it = ctx->tuned.find(key);
        if (it != ctx->tuned.end()) shape = it->second;
    }
    bool tuned_known = false;
    {
        std::lock_guard<std::mutex> tlk(ctx->tune_mu);
        tuned_known = ctx->tuned.count(key) > 0;
    }
    if (autotune && plan_hit && !tuned_known && cands.size() > 1) {
        float best = INFINITY;
        for (const Shape& c : cands) {
            float t = count_with(c, false);
            tuned_runs++;
            if (t < best) {
                best = t;
                shape = c;
            }
        }
        std::lock_guard<std::mutex> tlk(ctx->tune_mu);
        ctx->tuned[key] = shape;
    } else {
        // a batch's first count is launched directly (capturing costs more than
        // one replay gains); TPCF_PIPELINE=0 captures it at once
        const char* pl_env = getenv("TPCF_PIPELINE");
        count_with(shape, graphs && (plan_hit || (pl_env && pl_env[0] == '0')));
    }
    if (near && L.h_counters.p[CTR_DENSE]) {
        // a centre with more near tiles than a list holds: by tile triples, now
        // and whenever the batch comes again
        {
            std::lock_guard<std::mutex> tlk(ctx->tune_mu);
            if (ctx->refused.size() >= 65536) ctx->refused.clear();
            ctx->refused.insert(key);
        }
        run_group(ctx, L, group, false);
        return;
    }
    L.stats.tuned_shapes = tuned_runs;
    L.stats.hist_copies = (uint64_t)shape.copies;
    L.stats.ctas_per_sm = (uint64_t)shape.per_sm;
    float ms = 0, ms_main = 0;
    CK(cudaEventElapsedTime(&ms, L.ev0, L.ev1));
    CK(cudaEventElapsedTime(&ms_main, L.ev0, L.ev_mid));
    L.stats.main_kernel_ms = ms_main;
    // JBJ compat: the reference's two extra counts in bin 0 per visited triangle
    if (sp.kind == TPCF_TRIANGLE_JBJ && sp.overflow == TPCF_OVERFLOW_COMPAT && bin.len > 0 && part.begin == 0)
        for (size_t g = 0; g < group.size(); g++) L.h_hist.p[(size_t)bin.len * slot_of[g]] += 2 * job_units(g);
    for (size_t k = 0; k < nslots; k++) {
        const GroupJob& gj = group[slot_job[k]];
        const unsigned long long* src = L.h_hist.p + (size_t)bin.len * k;
        if (gj.accumulate) {
            for (int64_t b = 0; b < bin.len; b++) gj.out[b] += src[b];
        } else {
            memcpy(gj.out, src, (size_t)bin.len * sizeof(uint64_t));
        }
    }
    L.stats.graph_replays = replays;
    L.stats.kernel_ms = ms;
    L.stats.loop_units = units;
    // the fast triangle kernel skips (i,j) pairs that no counted triangle can
    // contain and counts the triangles it walks; the pair kernel counts the
    // pairs and tile pairs it finds; other kernels walk every triangle of
    // their units
    L.stats.evaluated_units = fast_tri || items ? dev_evaluated : header.evaluated;
    L.stats.binned_units = fast_tri ? dev_binned : L.stats.evaluated_units;
    L.stats.tasks = pairs ? dev_binned : near || tlist ? nrows : header.tiles;
    L.stats.kernel_launches = launches * std::max<uint64_t>(1, tuned_runs);
    L.stats.recheck_regrows = regrows;
    L.stats.total_ms =
        std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t_wall0).count();
    if (plan_trace()) {
        std::string line = "tpcf plan: jobs " + std::to_string(group.size()) + " rows " + std::to_string(nrows) +
                           " tiles " + std::to_string(L.stats.tasks) + " units " + std::to_string(header.nunits) +
                           " parts " + std::to_string(header.parts);
        double prev = 0;
        for (auto& ph : phases) {
            line += std::string(" ") + ph.first + " " + std::to_string(ph.second - prev);
            prev = ph.second;
        }
        line += " total " + std::to_string(L.stats.total_ms);
        fprintf(stderr, "%s\n", line.c_str());
    }
}

void add_stats(tpcf_stats& acc, const tpcf_stats& s) {
    acc.kernel_ms += s.kernel_ms;
    acc.main_kernel_ms += s.main_kernel_ms;
    acc.binned_units += s.binned_units;
    acc.total_ms += s.total_ms;
    acc.loop_units += s.loop_units;
    acc.evaluated_units += s.evaluated_units;
    acc.recheck_units += s.recheck_units;
    acc.recheck_regrows += s.recheck_regrows;
    acc.tasks += s.tasks;
    acc.kernel_launches += s.kernel_launches;
    acc.graph_replays += s.graph_replays;
    acc.plan_ms += s.plan_ms;
    acc.tuned_shapes += s.tuned_shapes;
    acc.hist_copies = s.hist_copies;
    acc.ctas_per_sm = s.ctas_per_sm;
}

// Counts a group: in one launch, or where its plan passes the limits in parts
// that add up -- the jobs in halves, a single job by ranges of its A tiles.
void count_group(tpcf_ctx* ctx, Lane& L, std::vector<GroupJob> group, bool lists = true, TileRange part = {}) {
    TooLarge e;
    try {
        run_group(ctx, L, group, lists, part);
        return;
    } catch (const TooLarge& x) {
        e = x;
    }
    if (group.size() == 1 && e.lists) return count_group(ctx, L, std::move(group), false);
    for (GroupJob& g : group)
        if (!g.accumulate) {
            int64_t len = 0;
            tpcf_hist_len(g.spec, &len);
            memset(g.out, 0, (size_t)len * sizeof(uint64_t));
            g.accumulate = true;
        }
    tpcf_stats acc{};
    auto half = [&](std::vector<GroupJob> jobs, TileRange r) {
        count_group(ctx, L, std::move(jobs), r.end < 0 && lists, r);
        add_stats(acc, L.stats);
    };
    if (group.size() > 1) {
        const auto mid = group.begin() + group.size() / 2;
        half({group.begin(), mid}, {});
        half({mid, group.end()}, {});
    } else {
        if (e.tiles < 2) throw InvalidArg{"too many tile triples in one batch"};
        const int mid = part.begin + e.tiles / 2;
        half(group, {part.begin, mid});
        half(group, {mid, part.begin + e.tiles});
    }
    L.stats = acc;
}

// before: a spec that passed (its value is not checked again), or null
void validate(const tpcf_spec* sp, const tpcf_job* job, const tpcf_spec* before = nullptr) {
    if (!sp || !job) throw InvalidArg{"null spec or job"};
    const bool flags_ok = (job->flags & ~(uint32_t)TPCF_JOB_GLOBAL_INDEX) == 0 && job->reserved == 0;
    if (before && flags_ok && memcmp(before, sp, sizeof *sp) == 0) return;
    if (sp->kind != TPCF_THREE_SIDE && sp->kind != TPCF_TRIANGLE && sp->kind != TPCF_PAIR &&
        sp->kind != TPCF_TRIANGLE_JBJ)
        throw InvalidArg{"bad kind"};
    if (sp->loop < TPCF_LOOP_ALL || sp->loop > TPCF_LOOP_ONE) throw InvalidArg{"bad loop"};
    if (sp->precision != TPCF_GUARDED_FP32 && sp->precision != TPCF_PLAIN_FP64 && sp->precision != TPCF_GEOMETRY_FP64)
        throw InvalidArg{"bad precision"};
    if (sp->precision == TPCF_GEOMETRY_FP64 && sp->kind != TPCF_TRIANGLE)
        throw InvalidArg{"TPCF_GEOMETRY_FP64 is implemented for the triangle parametrization only"};
    if (!flags_ok) throw InvalidArg{"bad job flags"};
    (void)make_binning(*sp);
}

template <typename F>
tpcf_status guarded(tpcf_ctx* ctx, F&& f) {
    try {
        f();
        return TPCF_OK;
    } catch (const InvalidArg& e) {
        return fail(ctx, TPCF_ERR_INVALID, e.msg);
    } catch (const InternalError& e) {
        return fail(ctx, TPCF_ERR_INTERNAL, e.msg);
    } catch (const CudaError& e) {
        cudaGetLastError();
        if (e.e == cudaErrorMemoryAllocation) return fail(ctx, TPCF_ERR_OOM, cudaGetErrorString(e.e));
        return fail(ctx, TPCF_ERR_CUDA, cudaGetErrorString(e.e));
    } catch (const std::bad_alloc&) {
        return fail(ctx, TPCF_ERR_OOM, "host allocation failed");
    } catch (...) {
        return fail(ctx, TPCF_ERR_INTERNAL, "unexpected exception");
    }
}

// footprint estimate of a job for admission (views are shared and cached)
int64_t job_bytes(tpcf_ctx* ctx, const tpcf_spec& sp, const tpcf_job& job) {
    int64_t b = 0;
    int nc = sp.kind == TPCF_PAIR ? 2 : 3;
    for (int r = 0; r < nc; r++) {
        auto it = ctx->catalogs.find(job.catalog[r]);
        if (it == ctx->catalogs.end()) continue;
        int64_t e = job.end[r] < 0 ? it->second->n : job.end[r];
        b += (e - job.begin[r]) * (int64_t)sizeof(float4);
    }
    int64_t len = 0;
    tpcf_hist_len(&sp, &len);
    return b + len * 8;
}

double now_ms() {
    return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now().time_since_epoch()).count();
}

// Serving worker on lane 'lane'.  It takes the oldest pending job plus every
// pending job of the same binning that fits the admission budget (device
// bytes of all batches in flight on the serving lanes), counts them in one
// persistent launch on its own stream and completes their tickets.  Jobs that
// arrive meanwhile are taken by the next free worker, so batches overlap on
// the device.
// Work estimate of a job for scheduling: the product of its catalog range
// sizes (the loop size up to a constant).
// Mean number of points of catalog range b within 'reach' of a point of range
// a, from 64 points spread over range a (cached per ranges and reach).
// Called with ctx->mu held.
double neighbour_density(tpcf_ctx* ctx, uint64_t ha, int64_t a0, int64_t a1, uint64_t hb, int64_t b0, int64_t b1,
                         double reach) {
    auto key = std::make_tuple(ha, a0, a1, hb, b0, b1, reach);
    auto hit = ctx->density.find(key);
    if (hit != ctx->density.end()) return hit->second;
    const Catalog& A = *ctx->catalogs.at(ha);
    const Catalog& B = *ctx->catalogs.at(hb);
    const int64_t na = a1 - a0;
    const double r2 = reach * reach;
    const int samples = (int)std::min<int64_t>(64, na);
    uint64_t near = 0;
    for (int t = 0; t < samples; t++) {
        const int64_t i = a0 + (int64_t)t * na / samples;
        for (int64_t j = b0; j < b1; j++) {
            const double dx = (double)A.x[i] - B.x[j], dy = (double)A.y[i] - B.y[j], dz = (double)A.z[i] - B.z[j];
            near += dx * dx + dy * dy + dz * dz < r2;
        }
    }
    const double rho = samples ? (double)near / samples : 0.0;
    ctx->density[key] = rho;
    return rho;
}

// Work estimate of a job for serving (which lane, how many per batch): the
// number of index pairs (pairs) or of i-j, i-k pairs of sides (triangles)
// within the largest side that can be counted, from the neighbour densities;
// the product of the range sizes where every triple counts.  Called with
// ctx->mu held, at submission.
double job_cost(tpcf_ctx* ctx, const tpcf_spec& sp, const tpcf_job& job) {
    int nc = sp.kind == TPCF_PAIR ? 2 : 3;
    int64_t b[3] = {0, 0, 0}, e[3] = {0, 0, 0};
    double prod = 1;
    for (int r = 0; r < nc; r++) {
        auto it = ctx->catalogs.find(job.catalog[r]);
        if (it == ctx->catalogs.end()) return 0;
        b[r] = job.begin[r];
        e[r] = job.end[r] < 0 ? it->second->n : job.end[r];
        prod *= (double)std::max<int64_t>(e[r] - b[r], 0);
    }
    const double reach = make_binning(sp).lmax;
    if (!(reach < 1e30) || (sp.kind == TPCF_THREE_SIDE && sp.overflow != TPCF_OVERFLOW_CLEAN)) return prod;
    const double na = (double)(e[0] - b[0]);
    double c = na * neighbour_density(ctx, job.catalog[0], b[0], e[0], job.catalog[1], b[1], e[1], reach);
    if (nc == 3) c *= neighbour_density(ctx, job.catalog[0], b[0], e[0], job.catalog[2], b[2], e[2], reach);
    return c;
}

void worker_loop(tpcf_ctx* ctx, int lane) {
    Lane& L = *ctx->lanes[lane];
    cudaSetDevice(ctx->device);
    // the first serving lane takes any job; the others only light ones, so
    // that light jobs keep flowing while heavy ones run
    const bool light_only = lane >= 2;
    auto heavy = [&](const Pending& p) { return p.cost > ctx->heavy_cost; };
    for (;;) {
        std::vector<std::shared_ptr<Pending>> batch;
        int64_t used = 0;
        {
            std::unique_lock<std::mutex> lk(ctx->qmu);
            for (;;) {
                ctx->qcv.wait(lk, [&] { return ctx->stop || !ctx->queue.empty(); });
                if (ctx->stop && ctx->queue.empty()) return;
                // drop cancelled jobs
                for (auto it = ctx->queue.begin(); it != ctx->queue.end();) {
                    if ((*it)->cancelled) {
                        (*it)->status = TPCF_ERR_CANCELLED;
                        (*it)->t_done = now_ms();
                        it = ctx->queue.erase(it);
                    } else {
                        ++it;
                    }
                }
                if (ctx->queue.empty()) continue;
                // the oldest job this lane takes
                std::shared_ptr<Pending> first;
                for (auto& p : ctx->queue)
                    if (!light_only || !heavy(*p)) {
                        first = p;
                        break;
                    }
                if (!first) {
                    ctx->qcv.wait(lk);
                    continue;
                }
                int64_t room = ctx->admit_bytes - ctx->inflight_bytes;
                int64_t fb = job_bytes(ctx, first->spec, first->job);
                // the oldest job waits for memory unless nothing else is in flight
                if (fb > room && ctx->inflight_bytes > 0) {
                    ctx->qcv.wait(lk);
                    continue;
                }
                // a heavy job runs alone; light jobs of the same binning share a
                // launch, up to a summed work estimate, so that a light batch
                // stays short and the jobs behind it start soon
                const bool first_heavy = heavy(*first);
                double batch_cost = 0;
                for (auto it = ctx->queue.begin(); it != ctx->queue.end();) {
                    auto& p = *it;
                    if (!same_binning(p->spec, first->spec) || p->spec.prune != first->spec.prune ||
                        (p != first && (first_heavy || heavy(*p)))) {
                        ++it;
                        continue;
                    }
                    const double c = p->cost;
                    if (!batch.empty() && batch_cost + c > ctx->light_batch_cost) break;
                    int64_t jb = job_bytes(ctx, p->spec, p->job);
                    if (!batch.empty() && used + jb > room) break;
                    used += jb;
                    batch_cost += c;
                    batch.push_back(p);
                    it = ctx->queue.erase(it);
                    if (batch.size() >= 4096) break;
                }
                // a heavy batch leaves SMs to the light lanes (its CTAs are persistent)
                L.sm_cap = first_heavy && ctx->reserve_sms > 0 ? ctx->num_sms - ctx->reserve_sms : 0;
                L.slice_batches = first_heavy && ctx->slice_heavy;
                ctx->inflight_bytes += used;
                break;
            }
        }
        ctx->qcv.notify_all();
        std::vector<GroupJob> group;
        int64_t len = 0;
        tpcf_hist_len(&batch[0]->spec, &len);
        double t_start = now_ms();
        for (auto& p : batch) {
            p->result.assign((size_t)len, 0);
            p->t_start = t_start;
            group.push_back({&p->spec, &p->job, p->result.data(), false});
        }
        tpcf_status st = guarded(ctx, [&] { count_group(ctx, L, group); });
        double t_done = now_ms();
        if (!ctx->trace_path.empty()) {
            double oldest = t_start;
            for (auto& p : batch) oldest = std::min(oldest, p->t_submit);
            char line[256];
            snprintf(line, sizeof(line), "%d %zu %llu %.3f %.3f %.3f %.3f\n", lane, batch.size(),
                     (unsigned long long)batch[0]->ticket, oldest, t_start, t_start + L.stats.plan_ms, t_done);
            std::lock_guard<std::mutex> lk(ctx->qmu);
            ctx->trace.push_back(line);
        }
        {
            std::lock_guard<std::mutex> lk(ctx->qmu);
            ctx->inflight_bytes -= used;
            for (auto& p : batch) {
                p->status = st;
                p->t_done = t_done;
            }
        }
        ctx->qcv.notify_all();
    }
}

}  // namespace

// ---------------------------------------------------------------------------
// C ABI

extern "C" {

int32_t tpcf_abi_version(void) { return TPCF_ABI_VERSION; }

const char* tpcf_status_string(tpcf_status s) {
    switch (s) {
        case TPCF_OK: return "ok";
        case TPCF_ERR_INVALID: return "invalid argument";
        case TPCF_ERR_CUDA: return "CUDA error";
        case TPCF_ERR_NO_DEVICE: return "no CUDA device";
        case TPCF_ERR_OOM: return "out of memory";
        case TPCF_ERR_TIMEOUT: return "timeout";
        case TPCF_ERR_NOT_FOUND: return "not found";
        case TPCF_ERR_CANCELLED: return "cancelled";
        case TPCF_ERR_INTERNAL: return "internal error";
        case TPCF_ERR_IO: return "I/O error";
        default: return "unknown status";
    }
}

const char* tpcf_last_error(tpcf_ctx* ctx) { return ctx ? ctx->last_error.c_str() : g_tls_error.c_str(); }

tpcf_status tpcf_create(tpcf_ctx** out, int32_t device) {
    if (!out) return fail(nullptr, TPCF_ERR_INVALID, "null output pointer");
    *out = nullptr;
    int count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess || count <= 0) {
        cudaGetLastError();
        return fail(nullptr, TPCF_ERR_NO_DEVICE, "no CUDA device visible");
    }
    if (device < 0 || device >= count) return fail(nullptr, TPCF_ERR_INVALID, "device index out of range");
    tpcf_ctx* ctx = new tpcf_ctx();
    tpcf_status s = guarded(ctx, [&] {
        ctx->device = device;
        CK(cudaSetDevice(device));
        CK(cudaDeviceGetAttribute(&ctx->num_sms, cudaDevAttrMultiProcessorCount, device));
        CK(cudaDeviceGetAttribute(&ctx->max_smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, device));
        CK(cudaDeviceGetAttribute(&ctx->max_smem_block, cudaDevAttrMaxSharedMemoryPerBlockOptin, device));
        CK(prepare_kernels(device));
        const char* tp = getenv("TPCF_TILE_POINTS");
        if (tp) ctx->tile_points = std::max(8, std::min(TILE, atoi(tp)));
        const char* adm = getenv("TPCF_ADMIT_BYTES");
        if (adm) ctx->admit_bytes = atoll(adm);
        const char* hc = getenv("TPCF_HEAVY_COST");
        if (hc) ctx->heavy_cost = atof(hc);
        if (const char* tr = getenv("TPCF_SERVING_TRACE")) ctx->trace_path = tr;
        if (const char* gt = getenv("TPCF_GROUP_TASKS")) ctx->group_tasks = std::min(MAX_WINDOW, std::max(1, atoi(gt)));
        const char* shv = getenv("TPCF_SLICE_HEAVY");
        if (shv) ctx->slice_heavy = shv[0] != '0';
        const char* stk = getenv("TPCF_SLICE_TASKS");
        if (stk) ctx->slice_tasks = std::max(0, atoi(stk));
        const char* lbc = getenv("TPCF_LIGHT_BATCH_COST");
        if (lbc) ctx->light_batch_cost = atof(lbc);
        // SMs a heavy serving batch leaves to the light lanes: none by default
        // (a quarter measured a higher p99 on the serving workload: the
        // heavy jobs themselves, slower, are the tail)
        const char* rs = getenv("TPCF_SERVING_RESERVE_SMS");
        if (rs) ctx->reserve_sms = std::max(0, std::min(ctx->num_sms - 1, atoi(rs)));
        const char* nw = getenv("TPCF_SERVING_LANES");
        int workers = nw ? std::max(1, std::min(8, atoi(nw))) : 3;
        for (int i = 0; i <= workers; i++) {
            auto L = std::make_unique<Lane>();
            // the light serving lanes (2 and up) get the highest stream
            // priority: their kernels start at the next slice boundary of a
            // heavy batch
            int prio_least = 0, prio_greatest = 0;
            CK(cudaDeviceGetStreamPriorityRange(&prio_least, &prio_greatest));
            CK(cudaStreamCreateWithPriority(&L->stream, cudaStreamNonBlocking, i >= 2 ? prio_greatest : prio_least));
            CK(cudaEventCreate(&L->ev0));
            CK(cudaEventCreate(&L->ev1));
            CK(cudaEventCreate(&L->ev_mid));
            if (i >= 1) {
                // serving lanes: buffers sized up front.  A device or
                // page-locked allocation issued while another lane's kernel
                // runs keeps this lane's next kernel from running beside it
                // (implicit synchronisation), so light batches must not allocate.
                L->h_hist.reserve((size_t)1 << 20);
                L->h_counters.reserve(CTR_WORDS);
                L->d_hist.reserve((size_t)1 << 22);
                L->d_counters.reserve(CTR_WORDS);
                // (three-side lists: per job of a batch of 4,096 its own, two
                // wedge jobs and an accumulator's; 32 MB of accumulators, as of
                // histograms)
                L->d_jobs.reserve((size_t)1 << 16);
                L->h_jobs.reserve((size_t)1 << 14);
                L->h_rows.reserve(((size_t)1 << 14) + 2);
                L->d_rows.reserve((size_t)1 << 16);
                L->d_acc.reserve((size_t)1 << 22);
                L->d_row_cnt.reserve((size_t)1 << 22);
                L->d_block_sum.reserve((size_t)1 << 17);
                L->d_units.reserve((size_t)1 << 20);
                L->d_masks.reserve((size_t)1 << 20);
                L->d_queue.reserve((size_t)1 << 22);
            }
            ctx->lanes.push_back(std::move(L));
        }
    });
    if (s != TPCF_OK) {
        g_tls_error = ctx->last_error;
        for (auto& L : ctx->lanes) L->release();
        delete ctx;
        return s;
    }
    for (size_t i = 1; i < ctx->lanes.size(); i++) ctx->workers.emplace_back(worker_loop, ctx, (int)i);
    *out = ctx;
    return TPCF_OK;
}

tpcf_status tpcf_destroy(tpcf_ctx* ctx) {
    if (!ctx) return TPCF_ERR_INVALID;
    {
        std::lock_guard<std::mutex> lk(ctx->qmu);
        ctx->stop = true;
    }
    ctx->qcv.notify_all();
    for (auto& t : ctx->workers)
        if (t.joinable()) t.join();
    if (!ctx->trace_path.empty()) {
        if (FILE* f = fopen(ctx->trace_path.c_str(), "w")) {
            for (auto& l : ctx->trace) fputs(l.c_str(), f);
            fclose(f);
        }
    }
    {
        std::lock_guard<std::recursive_mutex> lk(ctx->mu);
        std::lock_guard<std::recursive_mutex> vlk(ctx->view_mu);
        cudaSetDevice(ctx->device);
        for (auto& kv : ctx->pending_views) kv.second.fut.wait();
        ctx->pending_views.clear();
        ctx->views.clear();
        for (auto& L : ctx->lanes) L->release();
        ctx->acos_keys.release();
        ctx->acos_vals.release();
        ctx->acos_bucket.release();
    }
    delete ctx;
    return TPCF_OK;
}

tpcf_status tpcf_catalog_create(tpcf_ctx* ctx, const float* x, const float* y, const float* z, int64_t n,
                                uint64_t* handle) {
    if (!ctx || !handle || n < 0 || (n > 0 && (!x || !y || !z))) return fail(ctx, TPCF_ERR_INVALID, "bad catalog arguments");
    if (n > (int64_t)1 << 30) return fail(ctx, TPCF_ERR_INVALID, "catalog too large");
    std::lock_guard<std::recursive_mutex> lk(ctx->mu);
    return guarded(ctx, [&] {
        CK(cudaSetDevice(ctx->device));
        auto c = std::make_shared<Catalog>();
        c->n = n;
        c->x.assign(x, x + n);
        c->y.assign(y, y + n);
        c->z.assign(z, z + n);
        for (const std::vector<float>* v : {&c->x, &c->y, &c->z}) {
            bool ok = true;
            for (float f : *v) ok &= fabsf(f) <= 1e15f;
            c->tame = c->tame && ok;
        }
        std::lock_guard<std::recursive_mutex> vlk(ctx->view_mu);
        uint64_t h = ctx->next_handle++;
        ctx->catalogs[h] = c;
        // the resident form of a catalog is its spatial view (sorted points,
        // tiles, device copy), built on a thread of its own so that the
        // caller's next catalog (or anything else) proceeds meanwhile; the
        // first use waits for it.  Sub-range views are made on demand from the
        // host copy.
        const int dev = ctx->device, tile = ctx->tile_points;
        const uint64_t id = ++ctx->next_view_id;
        ctx->pending_views[std::make_tuple(h, (int64_t)0, n, tile, false)].id = id;
        ctx->pending_views[std::make_tuple(h, (int64_t)0, n, tile, false)].n = n;
        ctx->pending_views[std::make_tuple(h, (int64_t)0, n, tile, false)].fut =
            std::async(std::launch::async, [c, n, tile, dev, id] {
                CK(cudaSetDevice(dev));
                cudaStream_t st = nullptr;
                CK(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
                try {
                    auto v = build_view(*c, 0, n, tile, false, id, st);
                    cudaStreamDestroy(st);
                    return v;
                } catch (...) {
                    cudaStreamDestroy(st);
                    throw;
                }
            }).share();
        *handle = h;
    });
}

tpcf_status tpcf_catalog_release(tpcf_ctx* ctx, uint64_t handle) {
    if (!ctx) return TPCF_ERR_INVALID;
    std::lock_guard<std::recursive_mutex> vlk(ctx->view_mu);
    if (!ctx->catalogs.count(handle)) return fail(ctx, TPCF_ERR_NOT_FOUND, "unknown catalog handle");
    ctx->catalogs.erase(handle);
    for (auto it = ctx->views.begin(); it != ctx->views.end();) {
        if (std::get<0>(it->first) == handle) it = ctx->views.erase(it);
        else ++it;
    }
    // a view still being built: wait for it (its device buffers are freed
    // with the last reference), whatever its outcome
    for (auto it = ctx->pending_views.begin(); it != ctx->pending_views.end();) {
        if (std::get<0>(it->first) == handle) {
            it->second.fut.wait();
            it = ctx->pending_views.erase(it);
        } else {
            ++it;
        }
    }
    return TPCF_OK;
}

tpcf_status tpcf_resident_bytes(tpcf_ctx* ctx, int64_t* bytes) {
    if (!ctx || !bytes) return TPCF_ERR_INVALID;
    std::lock_guard<std::recursive_mutex> lk(ctx->view_mu);
    int64_t b = 0;
    for (auto& kv : ctx->views) b += (int64_t)kv.second->bytes();
    for (auto& kv : ctx->pending_views) {  // (a failed build holds nothing)
        try {
            b += (int64_t)kv.second.fut.get()->bytes();
        } catch (...) {
        }
    }
    *bytes = b;
    return TPCF_OK;
}

tpcf_status tpcf_hist_len(const tpcf_spec* sp, int64_t* len) {
    if (!sp || !len) return TPCF_ERR_INVALID;
    if (sp->kind == TPCF_THREE_SIDE) *len = (int64_t)sp->axis[0].nbins * sp->axis[0].nbins * sp->axis[0].nbins;
    else if (sp->kind == TPCF_TRIANGLE || sp->kind == TPCF_TRIANGLE_JBJ)
        *len = (int64_t)sp->axis[0].nbins * sp->axis[1].nbins * sp->axis[2].nbins;
    else if (sp->kind == TPCF_PAIR) *len = sp->axis[0].nbins;
    else return TPCF_ERR_INVALID;
    return TPCF_OK;
}

tpcf_status tpcf_loop_units(tpcf_ctx* ctx, const tpcf_spec* sp, const tpcf_job* job, uint64_t* units) {
    if (!ctx || !sp || !job || !units) return TPCF_ERR_INVALID;
    std::lock_guard<std::recursive_mutex> lk(ctx->view_mu);
    int64_t n[3] = {0, 0, 0};
    int nc = sp->kind == TPCF_PAIR ? 2 : 3;
    for (int r = 0; r < nc; r++) {
        auto it = ctx->catalogs.find(job->catalog[r]);
        if (it == ctx->catalogs.end()) return fail(ctx, TPCF_ERR_NOT_FOUND, "unknown catalog handle");
        int64_t e = job->end[r] < 0 ? it->second->n : job->end[r];
        n[r] = e - job->begin[r];
    }
    *units = loop_units(sp->kind, sp->loop, n);
    return TPCF_OK;
}

namespace {

// Jobs grouped by binning (and pruning); each group is one persistent launch.
// out_index == nullptr: job i writes hists[i]; else job i adds into
// hists[out_index[i]] (zeroed first).
tpcf_status count_jobs(tpcf_ctx* ctx, const tpcf_spec* specs, const tpcf_job* jobs, int32_t n,
                       const int32_t* out_index, int32_t n_out, uint64_t* const* hists) {
    std::lock_guard<std::recursive_mutex> lk(ctx->mu);
    return guarded(ctx, [&] {
        CK(cudaSetDevice(ctx->device));
        std::vector<int64_t> out_len(out_index ? n_out : 0, -1);
        for (int i = 0; i < n; i++) {
            validate(&specs[i], &jobs[i], i > 0 ? &specs[i - 1] : nullptr);
            if (out_index) {
                const int32_t o = out_index[i];
                if (o < 0 || o >= n_out) throw InvalidArg{"out_index out of range"};
                if (!hists[o]) throw InvalidArg{"null histogram pointer"};
                int64_t len = 0;
                tpcf_hist_len(&specs[i], &len);
                if (out_len[o] >= 0 && out_len[o] != len) throw InvalidArg{"jobs of one output differ in histogram length"};
                out_len[o] = len;
            } else if (!hists[i]) {
                throw InvalidArg{"null histogram pointer"};
            }
        }
        if (out_index)
            for (int32_t o = 0; o < n_out; o++)
                if (out_len[o] > 0) memset(hists[o], 0, (size_t)out_len[o] * sizeof(uint64_t));
        std::vector<char> done(n, 0);
        tpcf_stats acc{};
        for (int i = 0; i < n; i++) {
            if (done[i]) continue;
            std::vector<GroupJob> g;
            if (i == 0) g.reserve(n);
            for (int k = i; k < n; k++)
                if (!done[k] && same_binning(specs[k], specs[i]) && specs[k].prune == specs[i].prune) {
                    if (out_index) g.push_back({&specs[k], &jobs[k], hists[out_index[k]], true});
                    else g.push_back({&specs[k], &jobs[k], hists[k], false});
                    done[k] = 1;
                }
            Lane& L = *ctx->lanes[0];
            count_group(ctx, L, std::move(g));
            add_stats(acc, L.stats);
        }
        ctx->lanes[0]->stats = acc;
    });
}

}  // namespace

tpcf_status tpcf_count_batch(tpcf_ctx* ctx, const tpcf_spec* specs, const tpcf_job* jobs, int32_t n,
                             uint64_t* const* hists) {
    if (!ctx || !specs || !jobs || !hists || n < 0) return fail(ctx, TPCF_ERR_INVALID, "bad batch arguments");
    return count_jobs(ctx, specs, jobs, n, nullptr, 0, hists);
}

tpcf_status tpcf_count_batch_into(tpcf_ctx* ctx, const tpcf_spec* specs, const tpcf_job* jobs, int32_t n,
                                  const int32_t* out_index, int32_t n_out, uint64_t* const* hists) {
    if (!ctx || !specs || !jobs || !out_index || !hists || n < 0 || n_out < 0)
        return fail(ctx, TPCF_ERR_INVALID, "bad batch arguments");
    return count_jobs(ctx, specs, jobs, n, out_index, n_out, hists);
}

tpcf_status tpcf_convert_radecz(tpcf_ctx* ctx, const double* ra, const double* dec, const double* redshift,
                                int64_t n, const double* poly, float* x, float* y, float* z) {
    if (!ctx || n < 0 || (n > 0 && (!ra || !dec || !redshift || !x || !y || !z)))
        return fail(ctx, TPCF_ERR_INVALID, "bad conversion arguments");
    std::lock_guard<std::recursive_mutex> lk(ctx->mu);
    return guarded(ctx, [&] {
        if (n == 0) return;
        CK(cudaSetDevice(ctx->device));
        const double mice[3] = {-1.07199554e+00, 3.01313296e+03, -6.38827998e+02};  // the script's fit
        const double* pc = poly ? poly : mice;
        Lane& L = *ctx->lanes[0];
        DevBuf<double> d_in;
        DevBuf<float> d_out;
        d_in.reserve(3 * (size_t)n);
        d_out.reserve(3 * (size_t)n);
        const size_t b = (size_t)n * sizeof(double);
        CK(cudaMemcpyAsync(d_in.p, ra, b, cudaMemcpyHostToDevice, L.stream));
        CK(cudaMemcpyAsync(d_in.p + n, dec, b, cudaMemcpyHostToDevice, L.stream));
        CK(cudaMemcpyAsync(d_in.p + 2 * n, redshift, b, cudaMemcpyHostToDevice, L.stream));
        CK(launch_radecz_to_xyz(d_in.p, d_in.p + n, d_in.p + 2 * n, n, pc, d_out.p, d_out.p + n, d_out.p + 2 * n,
                                L.stream));
        const size_t fb = (size_t)n * sizeof(float);
        CK(cudaMemcpyAsync(x, d_out.p, fb, cudaMemcpyDeviceToHost, L.stream));
        CK(cudaMemcpyAsync(y, d_out.p + n, fb, cudaMemcpyDeviceToHost, L.stream));
        CK(cudaMemcpyAsync(z, d_out.p + 2 * n, fb, cudaMemcpyDeviceToHost, L.stream));
        CK(cudaStreamSynchronize(L.stream));
        L.h2d += 3 * b;
        L.d2h += 3 * fb;
    });
}

tpcf_status tpcf_count(tpcf_ctx* ctx, const tpcf_spec* spec, const tpcf_job* job, uint64_t* hist, int64_t hist_len) {
    if (!ctx || !spec || !job || !hist) return fail(ctx, TPCF_ERR_INVALID, "null argument");
    int64_t len = 0;
    if (tpcf_hist_len(spec, &len) != TPCF_OK || len != hist_len) return fail(ctx, TPCF_ERR_INVALID, "hist_len mismatch");
    uint64_t* hp[1] = {hist};
    return tpcf_count_batch(ctx, spec, job, 1, hp);
}

tpcf_status tpcf_submit(tpcf_ctx* ctx, const tpcf_spec* spec, const tpcf_job* job, uint64_t* ticket) {
    if (!ctx || !spec || !job || !ticket) return fail(ctx, TPCF_ERR_INVALID, "null argument");
    double cost = 0;
    tpcf_status s = guarded(ctx, [&] {
        std::lock_guard<std::recursive_mutex> lk(ctx->mu);
        validate(spec, job);
        int nc = spec->kind == TPCF_PAIR ? 2 : 3;
        for (int r = 0; r < nc; r++) {
            auto it = ctx->catalogs.find(job->catalog[r]);
            if (it == ctx->catalogs.end()) throw InvalidArg{"unknown catalog handle"};
            const int64_t e = job->end[r] < 0 ? it->second->n : job->end[r];
            if (job->begin[r] < 0 || job->begin[r] > e || e > it->second->n) throw InvalidArg{"catalog range out of bounds"};
        }
        cost = job_cost(ctx, *spec, *job);
    });
    if (s != TPCF_OK) return s;
    auto p = std::make_shared<Pending>();
    p->cost = cost;
    p->spec = *spec;
    p->job = *job;
    p->t_submit = now_ms();
    {
        std::lock_guard<std::mutex> lk(ctx->qmu);
        p->ticket = ctx->next_ticket++;
        ctx->queue.push_back(p);
        ctx->tickets[p->ticket] = p;
        *ticket = p->ticket;
    }
    ctx->qcv.notify_all();
    return TPCF_OK;
}

tpcf_status tpcf_wait_timed(tpcf_ctx* ctx, uint64_t ticket, uint64_t* hist, int64_t hist_len, int64_t timeout_ms,
                            double* latency_ms, double* run_ms) {
    if (!ctx) return TPCF_ERR_INVALID;
    std::unique_lock<std::mutex> lk(ctx->qmu);
    auto it = ctx->tickets.find(ticket);
    if (it == ctx->tickets.end()) return fail(ctx, TPCF_ERR_NOT_FOUND, "unknown ticket");
    auto p = it->second;
    auto ready = [&] { return p->status != 1; };
    if (timeout_ms < 0) ctx->qcv.wait(lk, ready);
    else if (!ctx->qcv.wait_for(lk, std::chrono::milliseconds(timeout_ms), ready)) return TPCF_ERR_TIMEOUT;
    ctx->tickets.erase(ticket);
    if (latency_ms) *latency_ms = p->t_done - p->t_submit;
    if (run_ms) *run_ms = p->t_start > 0 ? p->t_done - p->t_start : 0.0;
    if (p->status != TPCF_OK) return p->status;
    if (hist) {
        if ((int64_t)p->result.size() != hist_len) return fail(ctx, TPCF_ERR_INVALID, "hist_len mismatch");
        memcpy(hist, p->result.data(), p->result.size() * sizeof(uint64_t));
    }
    return TPCF_OK;
}

tpcf_status tpcf_wait(tpcf_ctx* ctx, uint64_t ticket, uint64_t* hist, int64_t hist_len, int64_t timeout_ms) {
    return tpcf_wait_timed(ctx, ticket, hist, hist_len, timeout_ms, nullptr, nullptr);
}

tpcf_status tpcf_cancel(tpcf_ctx* ctx, uint64_t ticket) {
    if (!ctx) return TPCF_ERR_INVALID;
    std::lock_guard<std::mutex> lk(ctx->qmu);
    auto it = ctx->tickets.find(ticket);
    if (it == ctx->tickets.end()) return TPCF_ERR_NOT_FOUND;
    if (it->second->status != 1) return TPCF_ERR_INVALID;  // already ran
    it->second->cancelled = true;
    for (auto q = ctx->queue.begin(); q != ctx->queue.end(); ++q)
        if ((*q)->ticket == ticket) {
            (*q)->status = TPCF_ERR_CANCELLED;
            ctx->queue.erase(q);
            break;
        }
    ctx->qcv.notify_all();
    return TPCF_OK;
}

tpcf_status tpcf_last_stats(tpcf_ctx* ctx, tpcf_stats* stats) {
    if (!ctx || !stats) return TPCF_ERR_INVALID;
    std::lock_guard<std::recursive_mutex> lk(ctx->mu);
    Lane& L = *ctx->lanes[0];
    *stats = L.stats;
    // byte counters cover everything copied since the previous stats read
    stats->h2d_bytes = L.h2d;
    stats->d2h_bytes = L.d2h;
    L.h2d = L.d2h = 0;
    return TPCF_OK;
}

// test hook (not in the public header): checks the device exception table
// against its own entries; returns the mismatch count or -1.
int64_t tpcf_debug_acos_selfcheck(tpcf_ctx* ctx, int64_t* table_size) {
    if (!ctx) return -1;
    std::lock_guard<std::recursive_mutex> lk(ctx->mu);
    int64_t r = -1;
    guarded(ctx, [&] {
        CK(cudaSetDevice(ctx->device));
        ensure_acos(ctx);
        DevBuf<unsigned int> mm;
        mm.reserve(1);
        CK(cudaMemset(mm.p, 0, 4));
        cudaStream_t st = ctx->lanes[0]->stream;
        CK(launch_acos_check(acos_table(ctx), 0, ctx->acos_n, mm.p, st));
        unsigned int h = 0;
        CK(cudaMemcpyAsync(&h, mm.p, 4, cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        r = h;
        if (table_size) *table_size = ctx->acos_n;
    });
    return r;
}

}  // extern "C"

// test hook (not in the public header): size and FNV-1a hash of this host's
// exact-acosf exception table (built or loaded from the cache; no GPU needed)
extern "C" int32_t tpcf_debug_acos_table_hash(uint64_t* n, uint64_t* hash) {
    AcosHost h = load_or_build_acos_table();
    uint64_t x = 1469598103934665603ull;
    for (size_t i = 0; i < h.keys.size(); i++) {
        x = (x ^ h.keys[i]) * 1099511628211ull;
        x = (x ^ h.vals[i]) * 1099511628211ull;
    }
    if (n) *n = h.keys.size();
    if (hash) *hash = x;
    return TPCF_OK;
}

// test hook (not in the public header): this host's exact-acosf exceptions as
// keys (float bits of c, sorted) and the direction (+1/-1 ulp) of glibc's value
// relative to (float)tpcf_acos_d(c).  Call with keys == NULL for the count.
extern "C" int32_t tpcf_debug_acos_exceptions(uint32_t* keys, int8_t* dir, uint64_t cap, uint64_t* n) {
    AcosHost h = load_or_build_acos_table();
    if (n) *n = h.keys.size();
    if (!keys || !dir) return TPCF_OK;
    for (size_t i = 0; i < h.keys.size() && i < cap; i++) {
        keys[i] = h.keys[i];
        int64_t d = (int64_t)h.vals[i] - (int64_t)fbits((float)tpcf_acos_d((double)ffrom(h.keys[i])));
        dir[i] = (int8_t)(d > 0 ? 1 : (d < 0 ? -1 : 0));
    }
    return TPCF_OK;
}

// test hook (not in the public header): replaces the context's exception table
// by the given one (e.g. another machine's glibc, to compare with files that
// machine produced).  dir: +1/-1 ulp relative to (float)tpcf_acos_d(c).
extern "C" int32_t tpcf_debug_set_acos_exceptions(tpcf_ctx* ctx, const uint32_t* keys, const int8_t* dir, uint64_t n) {
    if (!ctx || (n && (!keys || !dir))) return TPCF_ERR_INVALID;
    std::lock_guard<std::recursive_mutex> lk(ctx->mu);
    return guarded(ctx, [&] {
        CK(cudaSetDevice(ctx->device));
        AcosHost h;
        h.keys.assign(keys, keys + n);
        h.vals.resize(n);
        for (uint64_t i = 0; i < n; i++) {
            if (i && keys[i] <= keys[i - 1]) throw InvalidArg{"exception keys must be strictly increasing"};
            h.vals[i] = fbits((float)tpcf_acos_d((double)ffrom(keys[i]))) + (uint32_t)(int32_t)dir[i];
        }
        h.bucket.assign(65537, 0);
        size_t j = 0;
        for (uint32_t b = 0; b <= 65536; b++) {
            while (j < h.keys.size() && (h.keys[j] >> 16) < b) j++;
            h.bucket[b] = (uint32_t)j;
        }
        ctx->acos_n = (uint32_t)n;
        ctx->acos_keys.reserve(std::max<size_t>(n, 1));
        ctx->acos_vals.reserve(std::max<size_t>(n, 1));
        ctx->acos_bucket.reserve(65537);
        if (n) {
            CK(cudaMemcpy(ctx->acos_keys.p, h.keys.data(), n * 4, cudaMemcpyHostToDevice));
            CK(cudaMemcpy(ctx->acos_vals.p, h.vals.data(), n * 4, cudaMemcpyHostToDevice));
        }
        CK(cudaMemcpy(ctx->acos_bucket.p, h.bucket.data(), 65537 * 4, cudaMemcpyHostToDevice));
        ctx->acos_ready = true;
    });
}

// test hook (not in the public header): device blocks above `bytes` are refused
// as if memory had run out
extern "C" void tpcf_debug_alloc_limit(uint64_t bytes) { DeviceBlocks::get().set_limit((size_t)bytes); }

// test hook (not in the public header): device and page-locked blocks taken from
// the driver so far
extern "C" uint64_t tpcf_debug_allocations(void) { return g_allocations.load(); }
