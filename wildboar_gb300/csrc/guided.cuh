// guided.cuh -- FP64 distances on the cells a 32-bit sweep cannot rule out
// (guided.cu).
#pragma once

#include <algorithm>
#include <cstring>
#include <memory>

#include "elastic.cuh"

namespace wb {

// Output of a pair left to the full recurrence (a NaN payload no arithmetic
// produces).
constexpr long long kGuidedPending = 0x7ff8d7a05e1e57edLL;

// Kinds with a first pass that can leave pairs pending.
constexpr bool guided_kind(int kind) {
    return kind == K_DTW || kind == K_WDTW || kind == K_ADTW || kind == K_EDR || kind == K_LCSS;
}

struct GuidedPrep {
    long long lo, hi;            // order codes of the smallest / largest input
    unsigned long long queue;    // next tile of 32 pairs
    unsigned long long pending;  // pairs left to the full recurrence
    unsigned long long seen;     // pairs whose blocks were collected, and of them those
    unsigned long long heavy;    // left or with a fourth of their blocks
};

// Extremes of a series: fixed point, and the largest float magnitude.
struct GuidedRange {
    int lo, hi;
    float mag;
};

struct GuidedArgs {
    ElasticJob J;
    const float *xf = nullptr, *yf = nullptr;  // centred, scaled, padded float series
    const float *xl = nullptr, *yl = nullptr;  // their rests
    const int *xq = nullptr, *yq = nullptr;    // the same in fixed point
    const double *xd = nullptr, *yd = nullptr;  // the series as given
    int64_t xs = 0, ys = 0;                    // their strides
    const GuidedRange *xr = nullptr, *yr = nullptr;
    const float *wext = nullptr;  // wdtw: weight of i - j at woff + (j - i)
    int woff = 0;
    GuidedPrep *prep = nullptr;
    // Instead of the job's mode: items p, the pair of row p % rows.count and
    // column col0 + p / rows.count -- the `n_items` (device) ones of `items`,
    // or without it all p < n_all.
    const uint32_t *items = nullptr;
    const unsigned *n_items = nullptr;
    int64_t n_all = 0, col0 = 0;
    unsigned long long *left = nullptr;  // the job's pairs left over (ElasticJob)
    int64_t left_cap = 0, tail_cap = 0;
    unsigned need = 0;  // pairs seen before the kernel gives up
    // per resident thread, interleaved [...][thread]
    int64_t nth = 0;
    uint4 *ckrow = nullptr;   // [strip + 1][group of 4 columns] bottom rows
    uint4 *ckcol = nullptr;   // [strip][block][S / 4] last columns of the blocks
    // per resident thread, one after the other
    uint4 *list = nullptr;    // [block][word] collected blocks: position, mask (high, low)
    double *brow = nullptr;   // [2][column] FP64 bottom rows of two strips
    int groups = 0, blocks = 0, list_cap = 0, brow_cols = 0;
};

// Centred, scaled, padded copies of a job's series (guided.cu): floats and,
// where set, fixed point, the extremes of every series, extended weights.
struct GuidedSeries {
    float *xf = nullptr, *yf = nullptr;
    float *xl = nullptr, *yl = nullptr;  // the floats' rests
    int *xq = nullptr, *yq = nullptr;
    double *xd = nullptr, *yd = nullptr;  // the values as given, padded with 0
    int64_t xs = 0, ys = 0;  // strides; row series start at element 3
    GuidedRange *xr = nullptr, *yr = nullptr;
    float *wext = nullptr;
    int woff = 0, wlen = 0;
};
int guided_series(const ElasticJob &job, const GuidedSeries &out, GuidedPrep *prep,
                  cudaStream_t s);

// edr / lcss over the full band, bit-parallel (bit_edit.cu); *pending is null
// when it does not run, else the device counter of the pairs left.
bool bit_edit_supported(const ElasticJob &job);
size_t bit_edit_bytes(const ElasticJob &job);
int launch_bit_edit(const ElasticJob &job, Workspace &ws, size_t leave,
                    unsigned long long **pending);

// erp, msm and twe over the full band (elastic_wave.cu), the whole job in place
// of the ring or strip kernel.
bool wave_supported(const ElasticJob &job);
size_t wave_bytes(const ElasticJob &job);
int launch_wave(const ElasticJob &job, Workspace &ws);

// The guided evaluation in two steps, for a caller that runs it over several
// lists of pairs: buffers and float / fixed-point series of the job (the grid
// holds at most max_pairs pairs), then a run per list.  ctx.args.prep is null
// when the job cannot be guided.
struct GuidedContext {
    GuidedArgs args;
    int S = 8, grid = 0;
};
size_t guided_list_bytes(const ElasticJob &job, int64_t max_pairs);
int guided_prepare(const ElasticJob &job, Workspace &ws, size_t leave, int64_t max_pairs,
                   GuidedContext &ctx);
int guided_run(const GuidedContext &ctx, cudaStream_t s);

// Evaluates the job on what is left of the workspace beyond `leave` bytes and sets
// job.pending and job.left for the second pass; they stay null when the job is not
// guided (or too little is left).
int launch_guided(ElasticJob &job, Workspace &ws, size_t leave);

// argmin_distance of the dtw family over float32 bounds and guided
// evaluations (argmin_guided.cu).
bool argmin_guided_supported(const ElasticJob &job);
size_t argmin_guided_bytes(const ElasticJob &job);
// chunk boundaries of `ny` candidates for `nq` queries, from 0 to ny
std::vector<int64_t> argmin_guided_chunks(int64_t nq, int64_t ny, int64_t k);
class GuidedArgmin {
  public:
    int prepare(const ElasticJob &job, Workspace &ws, size_t leave, bool &ok);
    // sets job.pending for the second pass
    int launch_chunk(int index, const EaChunk &chunk, cudaStream_t s, ElasticJob &job);

  private:
    struct Impl;
    std::shared_ptr<Impl> impl_;
};

#ifdef __CUDACC__
#define WB_FLT_INF __int_as_float(0x7f800000)
#define WB_DBL_INF __longlong_as_double(0x7ff0000000000000LL)
#define WB_DBL_MAX 1.7976931348623157e308

// order-preserving integer code of a double (for atomicMin / atomicMax);
// NaN counts as infinite
__device__ __forceinline__ long long order_code(double v) {
    const long long b = __double_as_longlong(v);
    return b < 0 ? (long long)(0x8000000000000000ULL - (unsigned long long)b) : b;
}
__device__ __forceinline__ double order_value(long long c) {
    return __longlong_as_double(
        c < 0 ? (long long)(0x8000000000000000ULL - (unsigned long long)c) : c);
}

// Centre and power-of-two scale that map [lo, hi] into [-1, 1]; false where the
// values are not finite or too small.
__device__ __forceinline__ bool centre_scale(long long lo_code, long long hi_code,
                                             double &centre, double &scale) {
    const double lo = order_value(lo_code), hi = order_value(hi_code);
    const double half = hi * 0.5 - lo * 0.5;
    if (!(isfinite(lo) && isfinite(hi) && isfinite(half))) return false;
    centre = lo * 0.5 + hi * 0.5;
    const int e = half > 0.0 ? ilogb(half) + 1 : 0;
    // (FP64 sums of squares of smaller values would round at the subnormal
    // step, which the bounds do not cover)
    if (e < -400) return false;
    scale = scalbn(1.0, -e);
    return true;
}
__device__ __forceinline__ bool centre_scale(const GuidedPrep *prep, double &centre,
                                             double &scale) {
    return centre_scale(prep->lo, prep->hi, centre, scale);
}

__device__ __forceinline__ uint64_t pack2(float a, float b) {
    uint64_t p;
    asm("mov.b64 %0, {%1, %2};" : "=l"(p) : "f"(a), "f"(b));
    return p;
}

// bits k (k < 32) with 0 <= e - k < width: strip rows in band at a column,
// e = c - i0 - lo
__device__ __forceinline__ unsigned band_rows(int e, int width) {
    const unsigned upper = e < 0 ? 0u : (e >= 31 ? 0xffffffffu : (0xffffffffu >> (31 - e)));
    const int lb = e - width + 1;
    const unsigned lower = lb <= 0 ? 0u : (lb >= 32 ? 0xffffffffu : ((1u << lb) - 1u));
    return upper & ~lower;
}

// the band of every pair (all pairs of a job share it)
struct Band {
    int n, m, r, mx, mn, lo, width, ns;
    __device__ __forceinline__ Band(const ElasticJob &J, int S)
        : n(J.rows.len), m(J.cols.len), r(J.band), mx(imax(0, m - n) + r),
          mn(imax(0, n - m)), lo(-(mn + r - 1)), width(mx - lo), ns((n - 1 + S - 1) / S) {}
    // columns [cs, ce) of strip s (rows 1 + S s ...); s = -1: row 0
    __device__ __forceinline__ int cs(int s, int S) const {
        return imax(0, 1 + s * S - mn - r + 1);
    }
    __device__ __forceinline__ int ce(int s, int S) const {
        const int last = s < 0 ? 0 : imin(n - 1, s * S + S);
        return imin(m, last + mx);
    }
};

__device__ __forceinline__ bool is_pending(double v) {
    return __double_as_longlong(v) == kGuidedPending;
}
// Pair number q of the list of those left, and its output.
__device__ __forceinline__ double *left_pair(const ElasticJob &J, int64_t q, int64_t &rs,
                                             int64_t &cs) {
    const int64_t id = (int64_t)J.left[q];
    rs = cs = id;
    if (J.mode == PM_PAIRED) return J.out + rs;
    cs = id / J.rows.count;
    rs = id - cs * J.rows.count;
    return J.out + rs * J.out_ld + cs;
}
// This thread's number where the warps of all blocks come first, so that a few lists'
// worth of warps spread over the SMs.
__device__ __forceinline__ int64_t spread_lane() {
    const int64_t warp = (int64_t)(threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    return warp * 32 + (threadIdx.x & 31);
}
#endif

}  // namespace wb
