// subseq_dot.cu -- minimum euclidean and scaled euclidean subsequence
// distance with every window's distance bounded from float32 sliding dot
// products first.
//
// The reference sums (t - s)^2, or (s - (t - mean) / std)^2 with normalised
// shapelets, window by window in order and keeps the smallest sum and its
// first window (distance/_metric.pyx:561-682).  The same sums expand to
//   euclidean   sum t^2 + sum s^2 - 2 sum s t
//   scaled      sum s^2 + L - (2 / std) (sum s t' - mean' sum s),
// t' and mean' relative to a centre of the series (sum ((t - mean) / std)^2 = L for
// the window's own mean and std), so all windows of a series against all
// shapelets of one length are one sliding product: one fused multiply-add per
// (window, shapelet, value) instead of a subtraction, a multiply-add, an
// abandoning test and two loads.
//
// dot_filter_kernel: a block per (series, shapelets of one length).  A thread
// holds 8 consecutive windows x 4 shapelets; step k takes one new series value
// (the 8 values slide through registers) and one broadcast float4 of shapelet
// values for 32 multiply-adds.  The series lies in shared memory with one pad
// word per 8, which makes the lanes' stride of 8 conflict-free.  Bound: FP32
// multiply-adds.
//
// Error bound (u = 2^-24): inputs rounded once and L fused additions move a dot
// product by at most (L + 8) u sum |s t| <= (L + 8) u |s| |t|; the norms are
// summed in FP64; the float expression adds a few u of its terms.  For scaled
// windows |t'| = sqrt(L (std^2 + mean'^2)), and L stands for the normalised
// window's square sum, whose running sums are off by at most 4 T 2^-53 max t^2
// / std^2 (relative): windows with std^2 below 1e-5 max t^2 are not bounded but
// kept.  A window stays if its lower bound is at most the smallest upper bound;
// the others have a larger FP64 sum than the window of that bound.  The kept
// windows (1 per pair on random walks) are summed in FP64 with the reference's
// operations, a pair with more than kKeep of them goes through the FP64 scan.
//
// The scaled scan needs the reference's running sums of every window; they are
// stored as such (window_sums_kernel), and mean and standard deviation (a
// division and a root each) are formed for kept windows only.
//
// Measured on one GB300: 2000 z-normalised shapelets of 16 to 128 values x 400
// series of 1024: 158.5 ms (FP64 divisions per window tile and a float scan
// per shapelet) -> 9.9 ms, of which the filter takes 4.0, the running sums 1.0
// and the FP64 sums 1.4 ms; 10 000 shapelets x 1 000 series: 1.27 s -> 87 ms
// (with the shapelet values read through L1 instead of staged in shared memory
// the filter takes 4.8 ms).

#include <cfloat>

#include "guided.cuh"
#include "subseq.cuh"

namespace wb {

namespace {

constexpr int kThreads = 128;
constexpr int kWarps = kThreads / 32;
constexpr int kTile = 256;   // windows of a warp: 8 per lane
constexpr int kKeep = 8;     // windows kept per pair
constexpr int kCand = 48;    // candidates per shapelet before the final bound
constexpr int kMaxSeries = 8192;
constexpr int kUnitQuads = 16;
constexpr int kStaged = 512;  // shapelet values (x 4) in shared memory

struct Quad {  // up to 4 shapelets of one length
    int64_t first;  // position in `order`
    int64_t off;    // float4 offset of its values
    int count, len;
};
struct Unit {  // consecutive quads of one length
    int first, count, group, len;
};

struct Range {  // order codes of the smallest and largest value
    long long lo, hi;
};

struct DotArgs {
    SubseqJob J;
    const double *norm = nullptr;           // scaled: normalised shapelets (else J.shapelets)
    const double *ex = nullptr, *ex2 = nullptr;  // scaled: running sums per (group, series)
    const double *prefix = nullptr;         // euclidean: prefix sums of t'^2 per series
    const Quad *quads = nullptr;
    const Unit *units = nullptr;
    int n_units = 0;
    float4 *s4 = nullptr;                   // [quad][value] 4 shapelets' values
    float2 *sn = nullptr;                   // [4 quad + j]: sum s^2, sum s
    const float *xf = nullptr;              // t' of the series, stride x.len
    const float *xmax2 = nullptr;           // scaled: largest t^2 of the series (scaled units)
    const Range *range = nullptr;           // scaled: per series, euclidean: of everything
    uint32_t *windows = nullptr;            // [pair][kKeep]
    double *sums = nullptr;
    int *kept = nullptr;
    double *start = nullptr;                // euclidean: [pair] bound of the smallest sum
    uint32_t *extra = nullptr;
    unsigned *n_extra = nullptr;
};

// Smallest and largest value, one warp per row: scaled, of every series (the
// products' rounding counts against a window's deviation, so a series is centred
// by itself); euclidean, of the series and shapelets together.
template <bool SCALED>
__global__ void __launch_bounds__(256) dot_range_kernel(const SubseqJob J, Range *range) {
    double lo = WB_DBL_INF, hi = -WB_DBL_INF;
    auto reduce = [&](int64_t row) {
        long long l = order_code(lo), h = order_code(hi);
        for (int o = 16; o > 0; o >>= 1) {
            const long long l2 = __shfl_xor_sync(0xffffffffu, l, o);
            const long long h2 = __shfl_xor_sync(0xffffffffu, h, o);
            l = l2 < l ? l2 : l;
            h = h2 > h ? h2 : h;
        }
        if ((threadIdx.x & 31) != 0) return;
        if (SCALED) {
            range[row] = Range{l, h};
        } else {
            atomicMin(&range->lo, l);
            atomicMax(&range->hi, h);
        }
    };
    const int64_t total = J.x.count + (SCALED ? 0 : J.m);
    for (int64_t t = ((int64_t)blockIdx.x * 256 + threadIdx.x) >> 5; t < total;
         t += ((int64_t)gridDim.x * 256) >> 5) {
        const bool series = t < J.x.count;
        const double *src = series ? J.x.base + t * J.x.stride
                                   : J.shapelets + J.offsets[t - J.x.count];
        const int len = series ? J.x.len : (int)J.lengths[t - J.x.count];
        for (int i = threadIdx.x & 31; i < len; i += 32) {
            double v = src[i];
            if (isnan(v)) v = WB_DBL_INF;
            lo = v < lo ? v : lo;
            hi = v > hi ? v : hi;
        }
        if (SCALED) {
            reduce(t);
            lo = WB_DBL_INF;
            hi = -WB_DBL_INF;
        }
    }
    if (!SCALED) reduce(0);
}

// t' as floats; scaled: the largest t^2, euclidean: FP64 prefix sums of t'^2
// (by chunks of 32 with a warp scan).  One warp per series.
template <bool SCALED>
__global__ void __launch_bounds__(256)
dot_series_kernel(const SubseqJob J, const Range *range, float *xf, float *xmax2,
                  double *prefix) {
    const int lane = threadIdx.x & 31;
    for (int64_t s = ((int64_t)blockIdx.x * 256 + threadIdx.x) >> 5; s < J.x.count;
         s += ((int64_t)gridDim.x * 256) >> 5) {
        const Range R = range[SCALED ? s : 0];
        double centre = 0.0, scale = 1.0;
        centre_scale(R.lo, R.hi, centre, scale);
        const double *src = J.x.base + s * J.x.stride;
        float mx = 0.0f;
        double run = 0.0;
        for (int i0 = 0; i0 < J.x.len; i0 += 32) {
            const int i = i0 + lane;
            const double raw = i < J.x.len ? src[i] : 0.0;
            const double v = i < J.x.len ? (raw - centre) * scale : 0.0;
            if (i < J.x.len) xf[s * J.x.len + i] = (float)v;
            if (SCALED) {
                mx = fmaxf(mx, __double2float_ru(fabs(raw * scale)));
            } else {
                double p = v * v;
                for (int o = 1; o < 32; o <<= 1) {
                    const double q = __shfl_up_sync(0xffffffffu, p, o);
                    if (lane >= o) p += q;
                }
                p += run;
                if (i < J.x.len) prefix[s * (J.x.len + 1) + i + 1] = p;
                if (i == 0) prefix[s * (J.x.len + 1)] = 0.0;
                run = __shfl_sync(0xffffffffu, p, 31);
            }
        }
        if (SCALED) {
            for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            if (lane == 0) xmax2[s] = __fmul_ru(mx, mx);
        }
    }
}

// The running sums of scaled_euclidean_distance for every window of every
// (length group, series): ex, ex2 after adding the window's last value.
__global__ void __launch_bounds__(64)
window_sums_kernel(const SubseqJob J, double *ex_tab, double *ex2_tab) {
    const int64_t total = J.x.count * (int64_t)J.n_groups;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int g = (int)(t / J.x.count);
        const int64_t s = t - (int64_t)g * J.x.count;
        const int L = J.group_len[g];
        const double *T = J.x.base + s * J.x.stride;
        double *et = ex_tab + t * (int64_t)J.win_stride;
        double *e2t = ex2_tab + t * (int64_t)J.win_stride;
        double ex = 0, ex2 = 0;
        for (int i = 0; i < J.x.len; i++) {
            const double cv = T[i];
            ex = ex + cv;
            ex2 = ex2 + cv * cv;
            if (i >= L - 1) {
                const int w = i - L + 1;
                et[w] = ex;
                e2t[w] = ex2;
                const double old = T[w];
                ex = ex - old;
                ex2 = ex2 - old * old;
            }
        }
    }
}

// mean and std of a window from its running sums (scaled_euclidean_distance,
// distance/_metric.pyx:561-622)
__device__ __forceinline__ void window_stats(double ex, double ex2, int L, double &mean,
                                             double &sd) {
    mean = ex / (double)L;
    const double tmp = ex2 / (double)L - mean * mean;
    sd = tmp > 0 ? sqrt(tmp) : 1.0;
}

// running sums -> mean and std in place, for the FP64 scan of the rows (length
// group, series) with pairs left
__global__ void __launch_bounds__(256)
finish_stats_kernel(const SubseqJob J, double *ex_tab, double *ex2_tab,
                    const unsigned long long *redo, const unsigned char *redo_rows) {
    if (*redo == 0) return;
    for (int64_t row = blockIdx.x; row < J.x.count * (int64_t)J.n_groups; row += gridDim.x) {
        if (!redo_rows[row]) continue;
        const int L = J.group_len[row / J.x.count];
        double *ex = ex_tab + row * J.win_stride, *ex2 = ex2_tab + row * J.win_stride;
        for (int w = threadIdx.x; w <= J.x.len - L; w += 256) {
            double mean, sd;
            window_stats(ex[w], ex2[w], L, mean, sd);
            ex[w] = mean;
            ex2[w] = sd;
        }
    }
}

// one block per quad: 4 shapelets' values side by side (zeros up to a multiple
// of 8 values) and their sums
template <bool SCALED>
__global__ void __launch_bounds__(64) quad_kernel(const DotArgs A, int64_t n_quads) {
    const SubseqJob &J = A.J;
    const int lane = threadIdx.x & 31, half = threadIdx.x >> 5;
    double centre = 0.0, scale = 1.0;
    if (!SCALED) centre_scale(A.range->lo, A.range->hi, centre, scale);
    for (int64_t qd = blockIdx.x; qd < n_quads; qd += gridDim.x) {
        const Quad Q = A.quads[qd];
        const int len = (Q.len + 7) & ~7;
        float *dst = reinterpret_cast<float *>(A.s4 + Q.off);
        for (int j = half; j < 4; j += 2) {
            double ss = 0.0, sm = 0.0;
            const double *src = nullptr;
            if (j < Q.count)
                src = (SCALED ? A.norm : J.shapelets) + J.offsets[J.order[Q.first + j]];
            for (int k = lane; k < len; k += 32) {
                double v = 0.0;
                if (src && k < Q.len) v = SCALED ? src[k] : (src[k] - centre) * scale;
                dst[4 * k + j] = (float)v;
                ss += v * v;
                sm += v;
            }
            for (int o = 16; o > 0; o >>= 1) {
                ss += __shfl_xor_sync(0xffffffffu, ss, o);
                sm += __shfl_xor_sync(0xffffffffu, sm, o);
            }
            if (lane == 0) A.sn[4 * qd + j] = make_float2((float)ss, (float)sm);
        }
    }
}

__host__ __device__ __forceinline__ int padded(int i) { return i + (i >> 3); }
// Series values in shared memory: a tile's last lane reads up to
// kTile + 7 values past the series (zeros).
__host__ __device__ __forceinline__ int staged(int T) { return (T + kTile + 23) & ~7; }

// float -> unsigned preserving the order
__device__ __forceinline__ unsigned float_order(float f) {
    const unsigned u = __float_as_uint(f);
    return u & 0x80000000u ? ~u : u | 0x80000000u;
}
__device__ __forceinline__ float order_float(unsigned o) {
    return __uint_as_float(o & 0x80000000u ? o & 0x7fffffffu : ~o);
}

// Dot products of 8 windows (values from tp, padded) with 4 shapelets of Lp
// values at s4 (shared or global memory).
__device__ __forceinline__ void dot_tile(const float *tp, const float4 *s4, int Lp,
                                         float (&acc)[4][8]) {
    float tw[8];
#pragma unroll
    for (int i = 0; i < 8; i++) tw[i] = tp[i];
    tp += 9;  // the next 8 values
#pragma unroll 1
    for (int k = 0; k < Lp; k += 8) {
#pragma unroll
        for (int kk = 0; kk < 8; kk++) {
            const float4 s = s4[k + kk];
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const float v = tw[(kk + i) & 7];
                acc[0][i] = __fmaf_rn(s.x, v, acc[0][i]);
                acc[1][i] = __fmaf_rn(s.y, v, acc[1][i]);
                acc[2][i] = __fmaf_rn(s.z, v, acc[2][i]);
                acc[3][i] = __fmaf_rn(s.w, v, acc[3][i]);
            }
            tw[kk] = tp[kk];
        }
        tp += 9;
    }
}

template <bool SCALED>
__global__ void __launch_bounds__(kThreads, 5) dot_filter_kernel(const DotArgs A) {
    extern __shared__ float sm[];
    __shared__ float4 quad_s[kStaged];             // shapelet values of the slots' quads
    __shared__ unsigned best[kWarps][4];           // smallest upper bound, ordered
    __shared__ int n_cand[kWarps][4];
    __shared__ uint32_t cand_w[kWarps][4][kCand];
    __shared__ float cand_lo[kWarps][4][kCand];
    const unsigned FULL = 0xffffffffu;
    const SubseqJob &J = A.J;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int T = J.x.len;
    const int cols = padded(staged(T)) + 1;  // of the padded arrays
    float *ts = sm, *wb = sm + cols, *wm = sm + 2 * cols, *wf = sm + 3 * cols;
    for (int64_t b = blockIdx.x; b < J.x.count * (int64_t)A.n_units; b += gridDim.x) {
        const int64_t si = b / A.n_units;
        const Range R = A.range[SCALED ? si : 0];
        double centre = 0.0, scale = 1.0;
        if (!centre_scale(R.lo, R.hi, centre, scale)) continue;  // left to the FP64 scan
        const Unit U = A.units[b - si * A.n_units];
        const int L = U.len, nwin = T - L + 1;
        const int Lp = (L + 7) & ~7;
        __syncthreads();
        for (int i = threadIdx.x; i < staged(T); i += kThreads)
            ts[padded(i)] = i < T ? A.xf[si * T + i] : 0.0f;
        // constants of the windows: scaled (2 / std', 2 mean' / std',
        // |t'| / (std' sqrt(L))), euclidean (sum t'^2)
        const int64_t row = ((int64_t)U.group * J.x.count + si) * J.win_stride;
        bool open = false;  // one of the thread's windows is not bounded
        for (int w = threadIdx.x; w < nwin; w += kThreads) {
            const int p = padded(w);
            if constexpr (SCALED) {
                const double inv = 1.0 / (double)L;
                const double mean = A.ex[row + w] * inv;
                const double var = (A.ex2[row + w] * inv - mean * mean) * (scale * scale);
                const float vf = (float)var;
                const float mu = (float)((mean - centre) * scale);
                if (vf > __fmul_rn(1.1e-5f, A.xmax2[si]) && vf <= FLT_MAX) {
                    const float is = 1.0f / sqrtf(vf);
                    wb[p] = 2.0f * is;
                    wm[p] = 2.0f * is * mu;
                    wf[p] = sqrtf(1.0f + mu * is * mu * is) * 1.00001f;
                } else {  // not bounded
                    open = true;
                    wb[p] = 0.0f;
                    wm[p] = 0.0f;
                    wf[p] = 1e30f;
                }
            } else {
                const double *pre = A.prefix + si * (T + 1);
                wf[p] = (float)(pre[w + L] - pre[w]);
            }
        }
        // Windows without a bound stay in every pair (a flat stretch of the series,
        // or values far from 0): with more than kKeep of them the pairs go to the
        // scan whatever the products are.
        if (SCALED && __syncthreads_count(open) > kKeep) continue;
        float eabs = 0.0f;  // euclidean: rounding of the prefix sums
        if constexpr (!SCALED) eabs = __double2float_ru(A.prefix[si * (T + 1) + T] * 1e-11);
        const int tiles = (nwin + kTile - 1) / kTile;
        const int wpq = tiles >= 3 ? 4 : tiles;     // warps of one quad: 1, 2 or 4
        const int slots = kWarps / wpq, slot = wid / wpq, part = wid - slot * wpq;
        const int room = kStaged / slots;           // staged values of a quad
        for (int q0 = 0; q0 < U.count; q0 += slots) {
            const bool has = q0 + slot < U.count;
            const int64_t qd = U.first + (has ? q0 + slot : 0);
            __syncthreads();
            if (threadIdx.x < kWarps * 4) {
                best[threadIdx.x >> 2][threadIdx.x & 3] = 0xffffffffu;
                n_cand[threadIdx.x >> 2][threadIdx.x & 3] = 0;
            }
            const float4 *s4 = A.s4 + A.quads[qd].off;
            if (has && Lp <= room)
                for (int k = part * 32 + lane; k < Lp; k += wpq * 32) quad_s[slot * room + k] = s4[k];
            __syncthreads();
            float c0[4], c1[4], e1[4], e2[4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float2 n = A.sn[4 * qd + j];
                const float g = __fmul_ru((float)(L + 8), 6.2e-8f);
                if constexpr (SCALED) {
                    c0[j] = n.x + (float)L;
                    c1[j] = n.y;
                    e1[j] = 2e-6f * (n.x + (float)L) + 1e-30f;
                    e2[j] = 2.05f * g * sqrtf(n.x * (float)L);
                } else {
                    c0[j] = n.x;
                    e2[j] = g + 5e-7f;
                    e1[j] = e2[j] * n.x + eabs + 1e-30f;
                }
            }
            for (int t0 = 0; t0 < tiles; t0 += wpq) {
                const int w0 = (t0 + part) * kTile + 8 * lane;
                const bool run = has && t0 + part < tiles;
                float acc[4][8];
#pragma unroll
                for (int j = 0; j < 4; j++)
#pragma unroll
                    for (int i = 0; i < 8; i++) acc[j][i] = 0.0f;
                if (run) {
                    if (Lp <= room) dot_tile(ts + padded(w0), quad_s + slot * room, Lp, acc);
                    else dot_tile(ts + padded(w0), s4, Lp, acc);
                }
                // distances and bounds; acc becomes the lower bound
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    float up = WB_FLT_INF;
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        const int w = w0 + i, p = padded(w0) + i;
                        float lo = WB_FLT_INF;
                        if (run && w < nwin) {
                            float d, e;
                            if constexpr (SCALED) {
                                d = __fmaf_rn(-wb[p], acc[j][i], __fmaf_rn(wm[p], c1[j], c0[j]));
                                e = __fmaf_rn(e2[j], wf[p], e1[j]);
                            } else {
                                d = __fmaf_rn(-2.0f, acc[j][i], c0[j] + wf[p]);
                                e = __fmaf_rn(e2[j], wf[p], e1[j]);
                            }
                            lo = d - e;
                            up = fminf(up, d + e);
                        }
                        acc[j][i] = lo;
                    }
                    const unsigned u = __reduce_min_sync(FULL, float_order(up));
                    if (lane == 0 && run) atomicMin(&best[slot][j], u);
                }
                __syncthreads();
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const float limit = order_float(best[slot][j]);
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        if (acc[j][i] <= limit && run && w0 + i < nwin) {
                            const int at = atomicAdd(&n_cand[slot][j], 1);
                            if (at < kCand) {
                                cand_w[slot][j][at] = (uint32_t)(w0 + i);
                                cand_lo[slot][j][at] = acc[j][i];
                            }
                        }
                    }
                }
                __syncthreads();
            }
            // what the final bound leaves, up to kKeep windows per shapelet
            for (int j = part; j < 4; j += wpq) {
                const int count = A.quads[qd].count;
                if (!has || j >= count) continue;
                const int n = n_cand[slot][j];
                const float limit = order_float(best[slot][j]);
                const int64_t pair = si * J.m + J.order[A.quads[qd].first + j];
                int kept = 0;
                for (int c = 0; c < imin(n, kCand); c += 32) {
                    const bool in = c + lane < imin(n, kCand) && cand_lo[slot][j][c + lane] <= limit;
                    const unsigned mask = __ballot_sync(FULL, in);
                    const int at = kept + __popc(mask & ((1u << lane) - 1u));
                    if (in && at < kKeep) A.windows[pair * kKeep + at] = cand_w[slot][j][c + lane];
                    kept += __popc(mask);
                }
                if (n > kCand || kept > kKeep) kept = 0;
                if (lane == 0) {
                    if (!SCALED && limit < FLT_MAX)
                        A.start[pair] = (double)limit * 1.000001 / (scale * scale);
                    A.kept[pair] = kept;
                    if (kept > 1) {
                        const unsigned at = atomicAdd(A.n_extra, (unsigned)(kept - 1));
                        for (int c = 1; c < kept; c++)
                            A.extra[at + c - 1] = (uint32_t)(pair * kKeep + c);
                    }
                }
            }
        }
    }
}

// FP64 sums of the kept windows, a thread per window: first the pairs' first
// ones (a warp on one shapelet), then the few others.
template <bool SCALED>
__global__ void __launch_bounds__(128) dot_exact_kernel(const DotArgs A) {
    const SubseqJob &J = A.J;
    const int64_t per = (J.x.count + 31) / 32 * 32;
    const int64_t first = per * J.m, total = first + (int64_t)*A.n_extra;
    for (int64_t t = (int64_t)blockIdx.x * 128 + threadIdx.x; t < total;
         t += (int64_t)gridDim.x * 128) {
        int64_t sh, si, slot;
        if (t < first) {
            sh = J.order[t / per];
            si = t % per;
            if (si >= J.x.count) continue;
            slot = (si * J.m + sh) * kKeep;
        } else {
            slot = A.extra[t - first];
            si = slot / kKeep / J.m;
            sh = slot / kKeep - si * J.m;
        }
        if (A.kept[slot / kKeep] <= 0) continue;
        const int L = (int)J.lengths[sh];
        const int w = (int)A.windows[slot];
        const double *T = J.x.base + si * J.x.stride + w;
        double dist = 0.0;
        if constexpr (SCALED) {
            const double *S = A.norm + J.offsets[sh];
            const int64_t row = ((int64_t)J.group_of[sh] * J.x.count + si) * J.win_stride + w;
            double mean, sd;
            window_stats(A.ex[row], A.ex2[row], L, mean, sd);
            for (int k = 0; k < L; k++) {
                double x = __ldg(S + k);
                x = x - (T[k] - mean) / sd;
                dist = dist + x * x;
            }
        } else {
            const double *S = J.shapelets + J.offsets[sh];
            for (int k = 0; k < L; k++) {
                double x = T[k];
                x = x - __ldg(S + k);
                dist = dist + x * x;
            }
        }
        A.sums[slot] = dist;
    }
}

// smallest sum of each pair, the first window of equal ones; a pair without a
// finite one goes to the FP64 scan, which takes no window of an infinite sum
__global__ void __launch_bounds__(256)
dot_select_kernel(const DotArgs A, int64_t pairs, unsigned long long *redo,
                  unsigned char *redo_rows) {
    const int64_t pair = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (pair >= pairs) return;
    const int count = A.kept[pair];
    auto leave = [&]() {
        const int64_t si = pair / A.J.m;
        redo_rows[(int64_t)A.J.group_of[pair - si * A.J.m] * A.J.x.count + si] = 1;
        atomicAdd(redo, 1ull);
    };
    if (count <= 0) {
        leave();
        return;
    }
    double best = A.sums[pair * kKeep];
    uint32_t at = A.windows[pair * kKeep];
    for (int q = 1; q < count; q++) {
        const double d = A.sums[pair * kKeep + q];
        const uint32_t w = A.windows[pair * kKeep + q];
        if (d < best || (d == best && w < at)) {
            best = d;
            at = w;
        }
    }
    if (!(best < WB_DBL_INF)) {
        A.kept[pair] = 0;
        leave();
        return;
    }
    A.J.out_dist[pair] = sqrt(best);
    A.J.out_idx[pair] = at;
}

size_t dot_smem(int T) {
    return (size_t)4 * (padded(staged(T)) + 1) * sizeof(float);
}

}  // namespace

struct DotPlan {
    std::vector<Quad> quads;
    std::vector<Unit> units;
    int64_t s4 = 0;
};

// (the job's order, group_len and the host copy of the lengths in that order)
static void plan_quads(const std::vector<int64_t> &order, const std::vector<int64_t> &hlen,
                       const std::vector<int32_t> &group_of, DotPlan &P) {
    const int64_t m = (int64_t)order.size();
    for (int64_t t = 0; t < m;) {
        const int g = group_of[order[t]], len = (int)hlen[order[t]];
        int64_t u = t;
        while (u < m && group_of[order[u]] == g) u++;
        for (int64_t a = t; a < u;) {
            Unit U{(int)P.quads.size(), 0, g, len};
            for (; a < u && U.count < kUnitQuads; a += 4, U.count++) {
                P.quads.push_back(Quad{a, P.s4, (int)std::min<int64_t>(4, u - a), len});
                P.s4 += (len + 7) & ~7;
            }
            P.units.push_back(U);
        }
        t = u;
    }
}

bool subseq_dot_supported(const SubseqJob &J, bool scaled) {
    const int64_t pairs = J.x.count * J.m;
    // The filter's launches take 50 us more than the scan's where that has little to
    // do.  A scan's warp takes about 1 us for a value of a shapelet in its first
    // windows (FP64) and 12 ns in every further 32 (float, abandoned early): 20 x 100
    // of 30 x 300 values, 165 us so, 0.50 ms in all and 0.42 with the filter, 5 x 400,
    // 66 us, 0.42 and 0.42, 1 x 10 of 10 x 100, 10 us, 0.32 and 0.36.  (Scaled windows:
    // from the first on, 5 x 400 1.3 and 0.7 ms.)
    if (!scaled) {
        const double len = (double)J.total_values / (double)std::max<int64_t>(J.m, 1);
        const int64_t chunks = (J.m + J.chunk - 1) / J.chunk;
        const int64_t turns = 1 + J.x.count * chunks / (8 * device_info().sm_count);
        const double us = (double)((std::min<int64_t>(J.m, J.chunk) + 3) / 4 * turns) * len *
                          (1.0 + 0.012 * (J.x.len - len) / 32.0);
        if (us < 70.0) return false;
    }
    return !J.paired && J.x.len <= kMaxSeries && pairs < ((int64_t)1 << 31) / kKeep &&
           pairs * kKeep * 16 <= (int64_t)2 << 30;
}

size_t subseq_dot_bytes(const SubseqJob &J, bool scaled) {
    const int64_t pairs = J.x.count * J.m;
    // quads: at most one per shapelet, their values padded to 8
    return align256(J.m * sizeof(Quad)) + align256(J.m * sizeof(Unit)) +
           align256((J.total_values + 8 * J.m) * 16) + align256(J.m * 4 * sizeof(float2)) +
           align256(J.x.count * (int64_t)J.x.len * 4) + align256(J.x.count * 4) +
           (scaled ? 0 : align256(J.x.count * ((int64_t)J.x.len + 1) * 8) + align256(pairs * 8)) +
           align256(sizeof(GuidedPrep)) + align256((scaled ? J.x.count : 1) * sizeof(Range)) +
           align256(pairs * kKeep * 4) +
           align256(pairs * kKeep * 8) + align256(pairs * 4) +
           align256(pairs * (kKeep - 1) * 4) + align256(4) +
           align256(J.x.count * (int64_t)J.n_groups) + 4096;
}

int launch_subseq_dot(SubseqJob &J, bool scaled, const double *norm, double *ex, double *ex2,
                      const std::vector<int64_t> &order, const std::vector<int64_t> &hlen,
                      const std::vector<int32_t> &group_of, DotUploads &keep, Workspace &ws) {
    cudaStream_t s = ws.stream();
    const int64_t pairs = J.x.count * J.m;
    auto plan = std::make_shared<DotPlan>();
    plan_quads(order, hlen, group_of, *plan);
    keep.plan = plan;  // the uploads read it until the stream is synchronised
    const int64_t nq = (int64_t)plan->quads.size(), nu = (int64_t)plan->units.size();
    WB_TAKE(prep, GuidedPrep, ws, 1);
    WB_TAKE(range, Range, ws, scaled ? J.x.count : 1);
    WB_TAKE(quads, Quad, ws, nq);
    WB_TAKE(units, Unit, ws, nu);
    WB_TAKE(s4, float4, ws, plan->s4);
    WB_TAKE(sn, float2, ws, nq * 4);
    WB_TAKE(xf, float, ws, J.x.count * (int64_t)J.x.len);
    WB_TAKE(xmax2, float, ws, J.x.count);
    double *prefix = nullptr, *start = nullptr;
    if (!scaled) {
        prefix = ws.take<double>(J.x.count * ((int64_t)J.x.len + 1));
        start = ws.take<double>(pairs);
        if (!prefix || !start) return fail(WB_ENOMEM, "workspace reservation exceeded");
        WB_CUDA(cudaMemsetAsync(start, 0x7f, pairs * sizeof(double), s));  // 1.4e306
    }
    WB_TAKE(windows, uint32_t, ws, pairs * kKeep);
    WB_TAKE(sums, double, ws, pairs * kKeep);
    WB_TAKE(kept, int, ws, pairs);
    WB_TAKE(extra, uint32_t, ws, pairs * (kKeep - 1));
    WB_TAKE(n_extra, unsigned, ws, 1);
    const size_t rows_bytes = (size_t)J.x.count * J.n_groups;
    WB_TAKE(redo_rows, unsigned char, ws, rows_bytes);
    WB_CUDA(cudaMemcpyAsync(quads, plan->quads.data(), nq * sizeof(Quad), cudaMemcpyHostToDevice, s));
    WB_CUDA(cudaMemcpyAsync(units, plan->units.data(), nu * sizeof(Unit), cudaMemcpyHostToDevice, s));
    if (!scaled) {  // lo = a very large code, hi = a very small one
        WB_CUDA(cudaMemsetAsync(&range->lo, 0x7f, sizeof(range->lo), s));
        WB_CUDA(cudaMemsetAsync(&range->hi, 0x80, sizeof(range->hi), s));
    }
    WB_CUDA(cudaMemsetAsync(&prep->queue, 0, sizeof(prep->queue) + sizeof(prep->pending), s));
    WB_CUDA(cudaMemsetAsync(kept, 0, pairs * sizeof(int), s));
    WB_CUDA(cudaMemsetAsync(n_extra, 0, sizeof(unsigned), s));
    WB_CUDA(cudaMemsetAsync(redo_rows, 0, rows_bytes, s));
    DotArgs A;
    A.J = J;
    A.norm = norm;
    A.ex = ex;
    A.ex2 = ex2;
    A.prefix = prefix;
    A.quads = quads;
    A.units = units;
    A.n_units = (int)nu;
    A.s4 = s4;
    A.sn = sn;
    A.xf = xf;
    A.xmax2 = xmax2;
    A.range = range;
    A.windows = windows;
    A.sums = sums;
    A.kept = kept;
    A.start = start;
    A.extra = extra;
    A.n_extra = n_extra;
    const DeviceInfo &dev = device_info();
    const int64_t cap = (int64_t)dev.sm_count * 8;
    const int rows_grid = (int)std::min(cap, (J.x.count + J.m + 7) / 8);
    const int quad_grid = (int)std::min<int64_t>(nq, 65535);
    const size_t smem = dot_smem(J.x.len);
    auto run = [&](auto range_of, auto series, auto quad, auto filter, auto exact) -> int {
        range_of<<<rows_grid, 256, 0, s>>>(J, range);
        WB_LAUNCH_CHECK("dot_range_kernel");
        series<<<rows_grid, 256, 0, s>>>(J, range, xf, xmax2, prefix);
        WB_LAUNCH_CHECK("dot_series_kernel");
        quad<<<quad_grid, 64, 0, s>>>(A, nq);
        WB_LAUNCH_CHECK("quad_kernel");
        WB_CUDA(allow_shared(filter, smem));
        timer_begin("dot_filter_kernel", s);
        filter<<<(unsigned)std::min<int64_t>(J.x.count * nu, (int64_t)1 << 30), kThreads, smem, s>>>(A);
        timer_end(s);
        WB_LAUNCH_CHECK("dot_filter_kernel");
        const int64_t threads = (J.x.count + 31) / 32 * 32 * J.m;
        exact<<<(unsigned)std::min<int64_t>((threads + 127) / 128, (int64_t)dev.sm_count * 16), 128,
                0, s>>>(A);
        WB_LAUNCH_CHECK("dot_exact_kernel");
        return WB_OK;
    };
    if (scaled) {
        const int64_t rows = (int64_t)J.n_groups * J.x.count;
        window_sums_kernel<<<(unsigned)std::min<int64_t>((rows + 63) / 64, (int64_t)dev.sm_count * 32),
                             64, 0, s>>>(J, ex, ex2);
        WB_LAUNCH_CHECK("window_sums_kernel");
        WB_TRY(run(dot_range_kernel<true>, dot_series_kernel<true>, quad_kernel<true>,
                   dot_filter_kernel<true>, dot_exact_kernel<true>));
    } else {
        WB_TRY(run(dot_range_kernel<false>, dot_series_kernel<false>, quad_kernel<false>,
                   dot_filter_kernel<false>, dot_exact_kernel<false>));
    }
    dot_select_kernel<<<(unsigned)((pairs + 255) / 256), 256, 0, s>>>(A, pairs, &prep->pending,
                                                                      redo_rows);
    WB_LAUNCH_CHECK("dot_select_kernel");
    if (scaled) {
        finish_stats_kernel<<<dev.sm_count * 8, 256, 0, s>>>(J, ex, ex2, &prep->pending,
                                                             redo_rows);
        WB_LAUNCH_CHECK("finish_stats_kernel");
    }
    J.kept = kept;
    J.redo = &prep->pending;
    J.redo_rows = redo_rows;
    J.start = start;
    return WB_OK;
}

}  // namespace wb
