// bit_edit.cu -- edr and lcss over the full band as bit-parallel edit
// recurrences, exact.
//
// Both recurrences count: edr adds 0 or 1 per move, lcss adds 1 per match, and
// the FP64 values of the reference (edr_distance, lcss_distance,
// distance/_elastic.pyx:1437-1497, 1118-1183) are these integers.  With no
// band edge inside the matrix (whose neighbours read 0 in the reference) every
// difference between neighbouring cells is -1, 0 or 1 (edr) or 0 or 1 (lcss),
// so 32 rows of a column are a pair of words (edr: positive and negative
// vertical differences, Myers 1999 in the blocked form of Hyyro 2003; lcss: one
// word, Crochemore et al. 2001) and a column step takes about 17 (5)
// instructions for 32 cells.  The zero border of the reference is a zero
// difference everywhere.
//
// What is left is the match of each cell, |x_i - y_j| < eps (edr) or <= eps
// (lcss) on the reference's FP64 difference.  A float32 difference decides it
// unless it lies within its rounding bound of eps (about one cell in 10^6 on
// random walks); a column of 32 rows with such a cell is compared in FP64.  Per
// cell: subtract, subtract eps from the magnitude, shift the sign into the
// match word, half a 3-input minimum for the closest call.
//
// One thread per pair, 32 lanes share the column series (broadcast); strips of
// 32 rows in registers sweep all columns; a strip hands its bottom row's
// differences to the next as 1 (lcss) or 2 (edr) bits per column.  Bound: the
// instruction issue of the 3.5 instructions per cell of the match words.
// Measured on one GB300: edr eps = 1.6, 500 x 500 pairs of length 256: 101.7 ms
// (FP64 strips, 161 G cells/s) -> 3.1 ms (5.3 T cells/s).

#include <cstdlib>

#include "guided.cuh"

namespace wb {

namespace {

constexpr int kThreads = 128;

struct BitArgs {
    ElasticJob J;
    const float *xf = nullptr, *yf = nullptr;
    int64_t xs = 0, ys = 0;
    const GuidedRange *xr = nullptr, *yr = nullptr;
    GuidedPrep *prep = nullptr;
    uint2 *row = nullptr;  // [block of 32 columns][thread] bottom-row bits
    int64_t nth = 0;
};

// match word of rows i0 .. i0 + 31 in FP64 (row i0 in bit 0)
template <bool LCSS>
__device__ __noinline__ unsigned exact_matches(const double *X, int n, int i0, double y,
                                               long long eb) {
    unsigned eq = 0;
    for (int k = 0; k < 32; k++) {
        if (i0 + k >= n) break;
        const long long v = abs_bits(X[i0 + k] - y);
        if (LCSS ? v <= eb : v < eb) eq |= 1u << k;
    }
    return eq;
}

template <bool LCSS>
__global__ void __launch_bounds__(kThreads) bit_edit_kernel(const BitArgs A) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const ElasticJob &J = A.J;
    const int n = J.rows.len, m = J.cols.len;
    uint2 *row = A.row + (int64_t)blockIdx.x * kThreads + threadIdx.x;
    double centre = 0.0, scale = 1.0;
    const bool finite = centre_scale(A.prep, centre, scale);
    const int64_t chunks = (J.rows.count + 31) >> 5;
    const int64_t ntiles = J.mode == PM_PAIRED ? chunks : chunks * J.cols.count;
    for (;;) {
        unsigned long long t64 = 0;
        if (lane == 0) t64 = atomicAdd(&A.prep->queue, 1ull);
        const int64_t t = (int64_t)__shfl_sync(FULL, t64, 0);
        if (t >= ntiles) break;
        int64_t cs = t / chunks;
        int64_t rs = (t - cs * chunks) * 32 + lane;
        if (J.mode == PM_PAIRED) {
            rs = t * 32 + lane;
            cs = rs;
        }
        const bool active = rs < J.rows.count && !(J.mode == PM_UPPER && rs >= cs);
        if (!__any_sync(FULL, active)) continue;
        if (!active) {
            rs = J.rows.count - 1;
            cs = J.mode == PM_PAIRED ? rs : cs;
        }
        double eps = J.eps;
        if (!LCSS && J.std_rows) eps = cy_max(J.std_rows[rs], J.std_cols[cs]) / 4.0;
        const long long eb = eps_bits(eps);
        const float epsf = (float)(eps * scale);
        // |d~ - d| <= 2^-24 (|x| + |y| + |d|) and the rounding of eps and of
        // the last subtraction, doubled
        const float margin = __fmaf_ru(2.4e-7f, __fadd_ru(A.xr[rs].mag, A.yr[cs].mag),
                                       __fmaf_ru(2.4e-7f, fabsf(epsf), 1e-37f));
        const float *xr = A.xf + rs * A.xs + 3;
        const float *yr = A.yf + cs * A.ys;
        const double *X = J.rows.base + rs * J.rows.stride;
        const double *Y = J.cols.base + cs * J.cols.stride;
        int score = 0;
        for (int i0 = 0; finite && i0 < n; i0 += 32) {
            const bool last = i0 + 32 >= n;
            float x[32];
#pragma unroll
            for (int k = 0; k < 32; k++) x[k] = i0 + k < n ? xr[i0 + k] : WB_FLT_INF;
            unsigned pv = LCSS ? FULL : 0u, mv = 0u;
            for (int c0 = 0; c0 < m; c0 += 32) {
                uint2 in = make_uint2(0u, 0u), out = make_uint2(0u, 0u);
                uint2 *edge = row + (int64_t)(c0 >> 5) * A.nth;
                if (i0 > 0) in = *edge;
                const int cn = imin(32, m - c0);
#pragma unroll 1
                for (int c = 0; c < cn; c++) {
                    const float y = yr[c0 + c];
                    unsigned eq = 0;
                    float close = WB_FLT_INF;
#pragma unroll
                    for (int k = 31; k > 0; k -= 2) {
                        const float f1 = __fsub_rn(fabsf(__fsub_rn(x[k], y)), epsf);
                        const float f0 = __fsub_rn(fabsf(__fsub_rn(x[k - 1], y)), epsf);
                        eq = __funnelshift_l(__float_as_uint(f1), eq, 1);
                        eq = __funnelshift_l(__float_as_uint(f0), eq, 1);
                        asm("min.f32 %0, %1, %2, %3;"
                            : "=f"(close)
                            : "f"(close), "f"(fabsf(f1)), "f"(fabsf(f0)));
                    }
                    if (close <= margin) eq = exact_matches<LCSS>(X, n, i0, __ldg(Y + c0 + c), eb);
                    if constexpr (LCSS) {
                        const unsigned u = pv & eq;
                        const uint64_t sum = (uint64_t)pv + u + ((in.x >> c) & 1u);
                        pv = (unsigned)sum | (pv & ~eq);
                        out.x |= (unsigned)(sum >> 32) << c;
                    } else {
                        const unsigned hp = (in.x >> c) & 1u, hm = (in.y >> c) & 1u;
                        const unsigned xv = eq | mv;
                        eq |= hm;
                        const unsigned xh = (((eq & pv) + pv) ^ pv) | eq;
                        unsigned ph = mv | ~(xh | pv);
                        unsigned mh = pv & xh;
                        if (last) {
                            const int b = (n - 1) & 31;
                            score += (int)((ph >> b) & 1u) - (int)((mh >> b) & 1u);
                        }
                        out.x |= (ph >> 31) << c;
                        out.y |= (mh >> 31) << c;
                        ph = (ph << 1) | hp;
                        mh = (mh << 1) | hm;
                        pv = mh | ~(xv | ph);
                        mv = ph & xv;
                    }
                }
                *edge = out;
            }
            if (LCSS) score += __popc(~pv);
        }
        if (active) {
            double res = __longlong_as_double(kGuidedPending);
            if (finite)
                res = LCSS ? 1.0 - (double)score / (double)imin(J.len_norm_rows, J.len_norm_cols)
                           : (double)score / (double)imax(J.len_norm_rows, J.len_norm_cols);
            else
                atomicAdd(&A.prep->pending, 1ull);
            if (J.mode == PM_PAIRED) {
                J.out[rs] = res;
            } else {
                J.out[rs * J.out_ld + cs] = res;
                if (J.mode == PM_UPPER) J.out[cs * J.out_ld + rs] = res;
            }
        }
    }
}

struct Plan {
    int64_t xs, ys;
    int grid, words;
    size_t bytes;
};

Plan plan_bits(const ElasticJob &J) {
    Plan p;
    p.xs = ((int64_t)J.rows.len + 3 + 3) / 4 * 4;
    p.ys = ((int64_t)J.cols.len + 3) / 4 * 4;
    int nb = 0;
    if (J.kind == K_LCSS)
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, bit_edit_kernel<true>, kThreads, 0);
    else
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, bit_edit_kernel<false>, kThreads, 0);
    const int64_t chunks = (J.rows.count + 31) / 32;
    const int64_t want =
        ((J.mode == PM_PAIRED ? chunks : chunks * J.cols.count) * 32 + kThreads - 1) / kThreads;
    p.grid = (int)std::max<int64_t>(
        1, std::min<int64_t>(want, (int64_t)imax(nb, 1) * device_info().sm_count));
    p.words = (J.cols.len + 31) / 32;
    p.bytes = align256(J.rows.count * p.xs * 4) + align256(J.cols.count * p.ys * 4) +
              align256(J.rows.count * sizeof(GuidedRange)) +
              align256(J.cols.count * sizeof(GuidedRange)) + align256(sizeof(GuidedPrep)) +
              align256((size_t)p.grid * kThreads * p.words * sizeof(uint2)) + 4096;
    return p;
}

}  // namespace

// edr / lcss without a band edge inside the matrix
bool bit_edit_supported(const ElasticJob &J) {
    if (J.kind != K_EDR && J.kind != K_LCSS) return false;
    if (J.key || J.all_zero || J.pending) return false;
    if (J.mode == PM_UPPER && J.rows.count < 2) return false;  // no pairs
    const char *e = getenv("WB_GPU_ELASTIC");
    if (e && (strcmp(e, "ring") == 0 || strcmp(e, "strip") == 0)) return false;
    const int n = J.rows.len, m = J.cols.len;
    return imax(0, n - m) + J.band >= n && imax(0, m - n) + J.band >= m;
}

size_t bit_edit_bytes(const ElasticJob &J) {
    return bit_edit_supported(J) ? plan_bits(J).bytes : 0;
}

int launch_bit_edit(const ElasticJob &J, Workspace &ws, size_t leave,
                    unsigned long long **pending) {
    *pending = nullptr;
    const Plan p = plan_bits(J);
    if (ws.remaining() < p.bytes + leave) return WB_OK;
    cudaStream_t s = ws.stream();
    BitArgs A;
    A.J = J;
    A.xs = p.xs;
    A.ys = p.ys;
    A.nth = (int64_t)p.grid * kThreads;
    WB_TAKE(prep, GuidedPrep, ws, 1);
    WB_TAKE(xf, float, ws, J.rows.count * p.xs);
    WB_TAKE(yf, float, ws, J.cols.count * p.ys);
    WB_TAKE(xr, GuidedRange, ws, J.rows.count);
    WB_TAKE(yr, GuidedRange, ws, J.cols.count);
    WB_TAKE(row, uint2, ws, (size_t)A.nth * p.words);
    A.prep = prep;
    A.xf = xf;
    A.yf = yf;
    A.xr = xr;
    A.yr = yr;
    A.row = row;
    GuidedSeries S;
    S.xf = xf;
    S.yf = yf;
    S.xs = p.xs;
    S.ys = p.ys;
    S.xr = xr;
    S.yr = yr;
    WB_TRY(guided_series(J, S, prep, s));
    WB_CUDA(cudaMemsetAsync(&prep->queue, 0, sizeof(prep->queue) + sizeof(prep->pending), s));
    timer_begin("bit_edit_kernel", s);
    if (J.kind == K_LCSS) bit_edit_kernel<true><<<p.grid, kThreads, 0, s>>>(A);
    else bit_edit_kernel<false><<<p.grid, kThreads, 0, s>>>(A);
    timer_end(s);
    WB_LAUNCH_CHECK("bit_edit_kernel");
    *pending = &prep->pending;
    return WB_OK;
}

}  // namespace wb
