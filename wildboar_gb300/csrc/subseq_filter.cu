// subseq_filter.cu -- minimum dtw subsequence distance (dtw, ddtw) with a
// float32 sweep of every window in front of the FP64 recurrence.
//
// dtw_subsequence_distance (distance/_elastic.pyx:622-695) scans the windows
// of a series in order with early abandoning at the best distance so far and
// returns the smallest and its first window.  A window abandoned has a row
// minimum, hence (costs are not negative, rounding is monotone) a distance,
// above the best before it, so the result is the minimum over all windows, the
// first of equal ones.  Only windows whose distance can be that minimum need
// FP64.
//
// subseq_filter_kernel: one warp per (series, shapelet), one lane per window.
// A lane keeps the band of its last row in registers, aligned with the
// diagonal (cell k of row i is column i + k - (h - 1), h the half-width), so a
// cell is a subtraction, a 3-input minimum of B[k], B[k + 1] and the cell to
// the left, and a fused multiply-add, with one shared-memory read of the
// series (adjacent lanes, adjacent windows); the band needs no other memory.
// Every fourth row a warp whose row minima all lie above the bound gives up the
// 32 windows.  Bound: issue, 4 to 5 instructions per band cell.
//
// With A the float sum, e = 2^-24 (max|t| + max|s|) and g the roundings of at
// most 2 L + 16 operations, the FP64 distance d of a window satisfies
// (sqrt(A / (1 + g)) - e sqrt(2 L))^2 <= d <= (sqrt(A / (1 - g)) + e sqrt(2 L))^2;
// windows whose lower bound exceeds the smallest upper bound are dropped, the
// others (1 or 2 per pair on random walks) are kept per pair and evaluated by
// subseq_exact_kernel, a thread per window.  The 32 windows of a round are
// skipped where LB_Keogh (shapelet envelope over the band) already puts all of
// them above the bound.  A pair with more than kKeep of them
// (periodic or constant series) goes through the FP64 scan.
//
// Measured on one GB300: 200 shapelets of 16 to 128 values x 100 series of
// 1024, r = 0.1: 66.3 ms (FP64 scan) -> 2.6 ms (filter 1.2, FP64 0.6 ms;
// without LB_Keogh and with a thread per pair for the FP64 part 4.6 ms).

#include <cfloat>

#include "elastic_rec.cuh"
#include "guided.cuh"
#include "subseq_filter.cuh"

namespace wb {

namespace {

constexpr int kThreads = 128;
constexpr int kKeep = 8;       // windows kept per pair
constexpr int kMaxBlocks = 8;  // of 8 band cells in registers
constexpr int kPad = 8 * kMaxBlocks;
constexpr int kMaxSeries = 16384;  // in shared memory

struct FilterArgs {
    SubseqElasticJob J;
    const GuidedPrep *prep = nullptr;
    const float *xf = nullptr;   // series, stride J.x.len
    const float *sf = nullptr;   // packed shapelets
    const float *xmag = nullptr, *smag = nullptr;
    float2 *env = nullptr;        // packed: (min, max) of the shapelet over the band
    uint32_t *windows = nullptr;  // [pair][kKeep]
    double *sums = nullptr;       // [pair][kKeep] their FP64 sums
    int *kept = nullptr;          // [pair]
    double *start = nullptr;      // [pair] bound of the smallest sum, for the FP64 scan
    uint32_t *extra = nullptr;    // pair kKeep + q of the kept windows q >= 1
    unsigned *n_extra = nullptr;
    int per_block = 1;            // shapelets per block
};

// smallest and largest value of the series and shapelets; one warp per row
__global__ void __launch_bounds__(256)
filter_range_kernel(const SubseqElasticJob J, GuidedPrep *prep) {
    double lo = WB_DBL_INF, hi = -WB_DBL_INF;
    const int64_t total = J.x.count + J.m;
    for (int64_t t = ((int64_t)blockIdx.x * 256 + threadIdx.x) >> 5; t < total;
         t += ((int64_t)gridDim.x * 256) >> 5) {
        const bool series = t < J.x.count;
        const int64_t s = series ? t : t - J.x.count;
        const double *src = series ? J.x.base + s * J.x.stride : J.shp + J.off[s];
        const int len = series ? J.x.len : (int)J.len[s] - (J.slopes ? 2 : 0);
        for (int i = threadIdx.x & 31; i < len; i += 32) {
            double v = src[i];
            if (isnan(v)) v = WB_DBL_INF;
            lo = v < lo ? v : lo;
            hi = v > hi ? v : hi;
        }
    }
    long long l = order_code(lo), h = order_code(hi);
    for (int o = 16; o > 0; o >>= 1) {
        const long long l2 = __shfl_xor_sync(0xffffffffu, l, o);
        const long long h2 = __shfl_xor_sync(0xffffffffu, h, o);
        l = l2 < l ? l2 : l;
        h = h2 > h ? h2 : h;
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMin(&prep->lo, l);
        atomicMax(&prep->hi, h);
    }
}

// centred, scaled floats and their magnitudes; one warp per series / shapelet
__global__ void __launch_bounds__(256)
filter_convert_kernel(const SubseqElasticJob J, const GuidedPrep *prep, float *xf, float *sf,
                      float *xmag, float *smag) {
    const int lane = threadIdx.x & 31;
    double centre = 0.0, scale = 1.0;
    centre_scale(prep, centre, scale);
    const int64_t total = J.x.count + J.m;
    for (int64_t t = ((int64_t)blockIdx.x * 256 + threadIdx.x) >> 5; t < total;
         t += ((int64_t)gridDim.x * 256) >> 5) {
        const bool series = t < J.x.count;
        const int64_t s = series ? t : t - J.x.count;
        const double *src = series ? J.x.base + s * J.x.stride : J.shp + J.off[s];
        float *dst = series ? xf + s * J.x.len : sf + J.off[s];
        const int len = series ? J.x.len : (int)J.len[s] - (J.slopes ? 2 : 0);
        float mx = 0.0f;
        for (int i = lane; i < len; i += 32) {
            const float v = (float)((src[i] - centre) * scale);
            dst[i] = v;
            mx = fmaxf(mx, fabsf(v));
        }
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        if (lane == 0) (series ? xmag : smag)[s] = mx;
    }
}

// env[c]: extremes of the shapelet over the rows that column c may pair with
__global__ void __launch_bounds__(128) filter_envelope_kernel(const FilterArgs A) {
    const SubseqElasticJob &J = A.J;
    for (int64_t sh = blockIdx.x; sh < J.m; sh += gridDim.x) {
        const int L = (int)J.len[sh] - (J.slopes ? 2 : 0), h = J.band_of_len[sh];
        const float *s = A.sf + J.off[sh];
        for (int c = threadIdx.x; c < L; c += 128) {
            float lo = WB_FLT_INF, hi = -WB_FLT_INF;
            for (int i = imax(0, c - h + 1); i < imin(L, c + h); i++) {
                lo = fminf(lo, s[i]);
                hi = fmaxf(hi, s[i]);
            }
            A.env[J.off[sh] + c] = make_float2(lo, hi);
        }
    }
}

// LB_Keogh of the windows at t: false once no lane's sum is within the bound
__device__ __forceinline__ bool keogh_passes(const float2 *__restrict__ env, int L,
                                             const float *t, float bound) {
    float sum = 0.0f;
    for (int c = 0; c < L;) {
        const int stop = imin(L, c + 8);
        for (; c < stop; c++) {
            const float2 e = __ldg(env + c);
            const float d = fmaxf(fmaxf(__fsub_rn(t[c], e.y), __fsub_rn(e.x, t[c])), 0.0f);
            sum = __fmaf_rn(d, d, sum);
        }
        if (!__any_sync(0xffffffffu, sum <= bound)) return false;
    }
    return true;
}

// One row of the band: B holds row i - 1 on entry and row i on return.  t points
// at the value of cell 0's column.  `first` is the first cell with a column
// >= 0 (START: rows above h - 1), `width` the number of cells in band.
template <int NB, bool START>
__device__ __forceinline__ void band_row(float (&B)[8 * NB + 1], float x, const float *t,
                                         int first, int width) {
    float left = WB_FLT_INF;
#pragma unroll
    for (int k = 0; k < 8 * NB; k++) {
        const float d = __fsub_rn(x, t[k]);
        float best;
        asm("min.f32 %0, %1, %2, %3;" : "=f"(best) : "f"(B[k]), "f"(B[k + 1]), "f"(left));
        float v = __fmaf_rn(d, d, best);
        if (START) v = k >= first ? v : WB_FLT_INF;
        if (k >= 8 * NB - 8) v = k < width ? v : WB_FLT_INF;
        B[k] = v;
        left = v;
    }
}

// float dtw of shapelet s (L values, half-width h) with the window at t, or
// +inf once every lane's row minimum exceeds its bound
template <int NB>
__device__ float window_sum(const float *__restrict__ s, int L, int h, const float *t,
                            float bound) {
    const int width = 2 * h - 1;
    float B[8 * NB + 1];
#pragma unroll
    for (int k = 0; k <= 8 * NB; k++) B[k] = k == h - 1 ? 0.0f : WB_FLT_INF;
    const float *tc = t - (h - 1);
    int i = 0;
    const int start = imin(h - 1, L);
    for (; i < start; i++) band_row<NB, true>(B, __ldg(s + i), tc + i, h - 1 - i, width);
    while (i < L) {
        const int stop = imin(L, i + 4);
        for (; i < stop; i++) band_row<NB, false>(B, __ldg(s + i), tc + i, 0, width);
        float low = B[0];
#pragma unroll
        for (int k = 1; k < 8 * NB; k++) low = fminf(low, B[k]);
        if (!__any_sync(0xffffffffu, low <= bound)) return WB_FLT_INF;
    }
    float r = WB_FLT_INF;
#pragma unroll
    for (int k = 0; k < 8 * NB; k++)
        if (k == h - 1) r = B[k];
    return r;
}

__global__ void __launch_bounds__(kThreads) subseq_filter_kernel(const FilterArgs A) {
    extern __shared__ float sm[];
    __shared__ uint32_t keep_w[kThreads / 32][2 * kKeep + 32];
    __shared__ float keep_a[kThreads / 32][2 * kKeep + 32];
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const SubseqElasticJob &J = A.J;
    const int T = J.x.len;
    double centre = 0.0, scale = 1.0;
    if (!centre_scale(A.prep, centre, scale)) return;  // every pair is scanned in FP64
    const int64_t chunks = J.paired ? 1 : (J.m + A.per_block - 1) / A.per_block;
    float *ts = sm + kPad;
    for (int64_t b = blockIdx.x; b < J.x.count * chunks; b += gridDim.x) {
        const int64_t si = b / chunks;
        const int64_t s0 = J.paired ? si : (b - si * chunks) * A.per_block;
        const int64_t s1 = J.paired ? si + 1 : (s0 + A.per_block < J.m ? s0 + A.per_block : J.m);
        __syncthreads();
        for (int i = threadIdx.x - kPad; i < T + kPad; i += kThreads)
            ts[i] = i >= 0 && i < T ? A.xf[si * T + i] : 0.0f;
        __syncthreads();
        for (int64_t sh = s0 + wid; sh < s1; sh += kThreads / 32) {
            const int L = (int)J.len[sh] - (J.slopes ? 2 : 0);
            const int64_t pair = J.paired ? si : si * J.m + sh;
            if (J.slopes && L < 1) continue;  // left to the FP64 kernel
            const int h = J.band_of_len[sh];
            const int nwin = T - L + 1;
            const int nb = imin((2 * h - 1 + 7) / 8, kMaxBlocks + 1);
            if (nb > kMaxBlocks) continue;
            const float *s = A.sf + J.off[sh];
            const float K = 2.0f * (float)L;
            const float ek = __fmul_ru(
                __fmaf_ru(6.0e-8f, __fadd_ru(A.xmag[si], A.smag[sh]), 1e-37f), __fsqrt_ru(K));
            const float g = __fmul_ru(__fadd_ru(K, 16.0f), 6.2e-8f);
            // largest float sum a window may have beside one of sum a:
            // (sqrt(a) (1 + g) + 2 ek)^2 (1 + g), and an absolute term
            auto limit = [&](float a) {
                if (!(a < FLT_MAX)) return WB_FLT_INF;
                const float r = __fmaf_ru(2.0f, ek, __fmul_ru(__fsqrt_ru(a), __fadd_ru(1.000001f, g)));
                return __fadd_ru(__fmul_ru(__fmul_ru(r, r), __fadd_ru(1.000001f, g)), 1e-30f);
            };
            float bound = WB_FLT_INF;
            int n = 0;  // kept windows (uniform)
            bool full = false;
            for (int base = 0; base < nwin && !full; base += 32) {
                const int w = imin(base + lane, nwin - 1);
                // (the float sum is at least LB_Keogh's up to the roundings that
                // the bound allows for)
                if (bound < FLT_MAX && !keogh_passes(A.env + J.off[sh], L, ts + w, bound)) continue;
                float a;
                switch (nb) {
                    case 1: a = window_sum<1>(s, L, h, ts + w, bound); break;
                    case 2: a = window_sum<2>(s, L, h, ts + w, bound); break;
                    case 3: a = window_sum<3>(s, L, h, ts + w, bound); break;
                    case 4: a = window_sum<4>(s, L, h, ts + w, bound); break;
                    case 5: a = window_sum<5>(s, L, h, ts + w, bound); break;
                    case 6: a = window_sum<6>(s, L, h, ts + w, bound); break;
                    case 7: a = window_sum<7>(s, L, h, ts + w, bound); break;
                    default: a = window_sum<8>(s, L, h, ts + w, bound); break;
                }
                if (base + lane >= nwin) a = WB_FLT_INF;
                float low = a;
                for (int o = 16; o > 0; o >>= 1) low = fminf(low, __shfl_xor_sync(FULL, low, o));
                bound = fminf(bound, limit(low));
                unsigned mask = __ballot_sync(FULL, a <= bound && a < FLT_MAX);
                if (mask == 0) continue;
                if (n + __popc(mask) > 2 * kKeep) {  // drop what the new bound excludes
                    int kept = 0;
                    for (int q = 0; q < n; q++)
                        if (keep_a[wid][q] <= bound) {
                            if (lane == 0) {
                                keep_a[wid][kept] = keep_a[wid][q];
                                keep_w[wid][kept] = keep_w[wid][q];
                            }
                            __syncwarp();
                            kept++;
                        }
                    n = kept;
                    if (n + __popc(mask) > 2 * kKeep + 32) full = true;
                }
                if (!full) {
                    if ((mask >> lane) & 1u) {
                        const int at = n + __popc(mask & ((1u << lane) - 1u));
                        keep_a[wid][at] = a;
                        keep_w[wid][at] = (uint32_t)w;
                    }
                    n += __popc(mask);
                    __syncwarp();
                }
            }
            int count = 0;
            for (int q = 0; q < n && !full; q++)
                if (keep_a[wid][q] <= bound) {
                    if (lane == 0 && count < kKeep)
                        A.windows[pair * kKeep + count] = keep_w[wid][q];
                    count++;
                }
            __syncwarp();
            // 0: the FP64 scan takes the pair
            if (full || count > kKeep) count = 0;
            if (lane == 0) {
                // (`bound` is one of the smallest FP64 sum too, in scaled values)
                if (bound < FLT_MAX) A.start[pair] = (double)bound * 1.000001 / (scale * scale);
                A.kept[pair] = count;
                if (count > 1) {
                    const unsigned at = atomicAdd(A.n_extra, (unsigned)(count - 1));
                    for (int q = 1; q < count; q++) A.extra[at + q - 1] = (uint32_t)(pair * kKeep + q);
                }
            }
        }
    }
}

// FP64 sums of the kept windows, a thread per window: first the pairs' first
// windows (the threads of a warp on one shapelet), then the few others.
__global__ void __launch_bounds__(kThreads)
subseq_exact_kernel(const FilterArgs A, double *gring, int P) {
    const SubseqElasticJob &J = A.J;
    const int64_t gtid = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    const int64_t nth = (int64_t)gridDim.x * kThreads;
    RingG ring{gring + gtid, nth};
    const int64_t per = (J.x.count + 31) / 32 * 32;
    const int64_t first = J.paired ? per : per * J.m;
    const int64_t total = first + (int64_t)*A.n_extra;
    for (int64_t t = gtid; t < total; t += nth) {
        int64_t sh, si, slot;
        if (t < first) {
            sh = J.paired ? t : t / per;
            si = J.paired ? t : t - sh * per;
            if (si >= J.x.count) continue;
            slot = (J.paired ? si : si * J.m + sh) * kKeep;
        } else {
            slot = A.extra[t - first];
            const int64_t pair = slot / kKeep;
            si = J.paired ? pair : pair / J.m;
            sh = J.paired ? pair : pair - si * J.m;
        }
        if (A.kept[slot / kKeep] <= 0) continue;
        const int L = (int)J.len[sh] - (J.slopes ? 2 : 0);
        double key;
        A.sums[slot] = rec_dtw<false>(ring, P, J.shp + J.off[sh], L,
                                      J.x.base + si * J.x.stride + A.windows[slot], L,
                                      J.band_of_len[sh], nullptr, key);
    }
}

// the smallest sum of each pair, the first window of equal ones; a pair without
// a finite one goes to the FP64 scan, which takes no window of an infinite sum
__global__ void __launch_bounds__(256)
subseq_select_kernel(const FilterArgs A, int64_t pairs, unsigned long long *redo) {
    const int64_t pair = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (pair >= pairs) return;
    const int count = A.kept[pair];
    if (count <= 0) {
        atomicAdd(redo, 1ull);
        return;
    }
    double best = A.sums[pair * kKeep];
    uint32_t at = A.windows[pair * kKeep];
    for (int q = 1; q < count; q++)
        if (A.sums[pair * kKeep + q] < best) {
            best = A.sums[pair * kKeep + q];
            at = A.windows[pair * kKeep + q];
        }
    if (!(best < WB_DBL_INF)) {
        A.kept[pair] = 0;
        atomicAdd(redo, 1ull);
        return;
    }
    A.J.out_dist[pair] = sqrt(best);
    A.J.out_idx[pair] = at;
}

int64_t pairs_of(const SubseqElasticJob &J) { return J.paired ? J.x.count : J.x.count * J.m; }

}  // namespace

bool subseq_filter_supported(const SubseqElasticJob &J, int kind, int max_band, int64_t total) {
    // The filter's launches take 35 us more than the scan's where that has little to
    // do: band cells of 32 windows that a scan's warp evaluates, 330 cycles each (1 x
    // 10 of 10 and 100 values, 40 cells, 0.33 ms, with the filter 0.36; 5 x 400 of 30 and
    // 300, 1350 cells, 0.89 and 0.46).
    const int64_t len = total / std::max<int64_t>(J.m, 1);
    const int64_t turns = 1 + pairs_of(J) / (16 * device_info().sm_count);
    if ((J.x.len - len) / 32 * len * (2 * max_band - 1) * turns < 200) return false;
    return kind == K_DTW && !J.prof_raw && J.x.len <= kMaxSeries &&
           2 * max_band - 1 <= 8 * kMaxBlocks && pairs_of(J) < ((int64_t)1 << 31) / kKeep &&
           pairs_of(J) * kKeep * 16 <= (int64_t)2 << 30;
}

size_t subseq_filter_bytes(const SubseqElasticJob &J, int64_t total) {
    const int64_t pairs = pairs_of(J);
    return align256(J.x.count * (int64_t)J.x.len * 4) + align256(total * 4) +
           align256(J.x.count * 4) + align256(J.m * 4) + align256(total * 8) +
           align256(pairs * kKeep * 4) + align256(pairs * kKeep * 8) +
           align256(pairs * (kKeep - 1) * 4) + 2 * align256(pairs * 4 + 4) +
           align256(pairs * 8) +
           align256(sizeof(GuidedPrep)) + 4096;
}

int launch_subseq_filter(SubseqElasticJob &J, int64_t total, double *gring, int P, int grid,
                         Workspace &ws, cudaStream_t s) {
    const int64_t pairs = pairs_of(J);
    FilterArgs A;
    WB_TAKE(prep, GuidedPrep, ws, 1);
    WB_TAKE(xf, float, ws, J.x.count * (int64_t)J.x.len);
    WB_TAKE(sf, float, ws, total);
    WB_TAKE(xmag, float, ws, J.x.count);
    WB_TAKE(smag, float, ws, J.m);
    WB_TAKE(windows, uint32_t, ws, pairs * kKeep);
    WB_TAKE(kept, int, ws, pairs);
    WB_TAKE(env, float2, ws, total);
    WB_TAKE(sums, double, ws, pairs * kKeep);
    WB_TAKE(extra, uint32_t, ws, pairs * (kKeep - 1));
    WB_TAKE(n_extra, unsigned, ws, 1);
    WB_TAKE(start, double, ws, pairs);
    A.J = J;
    A.prep = prep;
    A.xf = xf;
    A.sf = sf;
    A.xmag = xmag;
    A.smag = smag;
    A.windows = windows;
    A.kept = kept;
    A.env = env;
    A.sums = sums;
    A.extra = extra;
    A.n_extra = n_extra;
    A.start = start;
    const DeviceInfo &dev = device_info();
    const int64_t cap = (int64_t)dev.sm_count * 4;
    WB_CUDA(cudaMemsetAsync(&prep->lo, 0x7f, sizeof(prep->lo), s));
    WB_CUDA(cudaMemsetAsync(&prep->hi, 0x80, sizeof(prep->hi), s));
    WB_CUDA(cudaMemsetAsync(&prep->queue, 0, sizeof(prep->queue) + sizeof(prep->pending), s));
    WB_CUDA(cudaMemsetAsync(kept, 0, pairs * sizeof(int), s));
    WB_CUDA(cudaMemsetAsync(start, 0x7f, pairs * sizeof(double), s));  // 1.4e306
    WB_CUDA(cudaMemsetAsync(n_extra, 0, sizeof(unsigned), s));
    const int prep_grid = (int)std::min(cap, (J.x.count + J.m + 7) / 8);
    filter_range_kernel<<<prep_grid, 256, 0, s>>>(J, prep);
    WB_LAUNCH_CHECK("filter_range_kernel");
    filter_convert_kernel<<<prep_grid, 256, 0, s>>>(J, prep, xf, sf, xmag, smag);
    WB_LAUNCH_CHECK("filter_convert_kernel");
    filter_envelope_kernel<<<(int)std::min<int64_t>(J.m, 65535), 128, 0, s>>>(A);
    WB_LAUNCH_CHECK("filter_envelope_kernel");
    // a block stages its series once for its shapelets; fewer shapelets per
    // block where there would be too few blocks for the SMs
    const int64_t want = (int64_t)dev.sm_count * 32;
    const int64_t m = J.paired ? 1 : J.m;
    A.per_block = (int)std::max<int64_t>(
        4, std::min<int64_t>(64, J.x.count * m / std::max<int64_t>(want, 1)));
    const int64_t blocks = J.x.count * ((m + A.per_block - 1) / A.per_block);
    const size_t smem = (size_t)(J.x.len + 2 * kPad) * sizeof(float);
    WB_CUDA(allow_shared(subseq_filter_kernel, smem));
    timer_begin("subseq_filter_kernel", s);
    subseq_filter_kernel<<<(unsigned)std::min<int64_t>(blocks, (int64_t)1 << 30), kThreads, smem,
                           s>>>(A);
    timer_end(s);
    WB_LAUNCH_CHECK("subseq_filter_kernel");
    subseq_exact_kernel<<<grid, kThreads, 0, s>>>(A, gring, P);
    WB_LAUNCH_CHECK("subseq_exact_kernel");
    subseq_select_kernel<<<(unsigned)((pairs + 255) / 256), 256, 0, s>>>(A, pairs, &prep->pending);
    WB_LAUNCH_CHECK("subseq_select_kernel");
    J.kept = kept;
    J.redo = &prep->pending;
    J.start = start;
    return WB_OK;
}

}  // namespace wb
