// elastic_wave.cu -- erp, msm and twe over the full band: strips of a pair
// spread over the lanes of a warp.
//
// With no band edge inside the matrix a strip of kRows rows needs only the
// bottom row of the strip above it, one column later.  G = 1, 2, 4, .. 32 lanes
// share a pair: lane g sweeps strips g, g + G, .., one column per step and one
// column behind lane g - 1, whose bottom cell it takes by shuffle; lane 0 takes
// it from a row in global memory that lane G - 1 writes.  The operations of a
// cell and their order are those of the strip kernel (elastic_strip.cu), so the
// results are the reference's bits (erp_distance, msm_distance, twe_distance,
// distance/_elastic.pyx:1530-1580, 1592-1647, 1860-1921).
//
// Bound: the FP64 pipe, 18.7 cycles of an SM per warp instruction and 71 cycles
// of latency that the warp waits for.  So
//   * warps: one block per warp and the same number of pairs for every group of
//     lanes, so that the SMs get equal shares; G is the one with the least
//     steps x hypot(latency of a step, its FP64 time x warps of an SM);
//   * operations: msm 7.8 FP64 instructions a cell -> 4.3.  c + |x_i - y_j| is
//     formed once for both moves, c + |x_i - x_{i-1}| once per row and c +
//     |y_j - y_{j-1}| once per column (c + min(a, b) == min(c + a, c + b), the
//     rounding being monotone), on the integer and FP32 pipes; twe 8 -> 7:
//     |x_{i-1} - y_{j-1}| is the previous diagonal cell's |x_i - y_j|, and the
//     stiffness of a diagonal moves down a strip instead of being loaded (200 x
//     150 pairs of 256 34.1 -> 32.4 ms).
// With one lane per pair the last strip evaluates its own rows only (with G > 1 the
// lanes of a warp are at different strips, which would run one after the other):
// erp, 700 x 700 pairs of 57 (8 strips, the last of 1 row) 15.4 -> 13.9 ms, msm, 400
// x 400 of 60 6.7 -> 5.6.
// Measured on one GB300 against the strip and ring kernels (one thread per
// pair, whose busiest SM had 1.27 times the mean): msm, 301 x 290 pairs of 256 x
// 250 111.7 -> 48.6 ms (44 ms of FP64 instructions), 9 x 10 of 256 26.2 ->
// 0.94 ms; twe, 20 x 20 of 500 95.8 -> 3.0 ms; erp, 200 x 150 of 256 20.9 -> 16.9
// ms.

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <type_traits>

#include "guided.cuh"

namespace wb {

namespace {

constexpr int kRows = 8;

// c + f rounded to double as the FP64 pipe does it, for floats c, f >= 0.
// The float sum s and its error e are exact together (Dekker 1971), and the
// double nearest to s + e is s moved by e in units of the doubles' spacing at
// s, rounded to nearest even: s is an even number of units, and consecutive
// doubles have consecutive patterns.  Below a power of two the spacing is half.
__device__ __forceinline__ double add_nonneg(float c, float f) {
    const float s = __fadd_rn(c, f);
    const unsigned u = __float_as_uint(s);
    // s < 2^-74 (the unit's reciprocal is no float), infinite or NaN
    if (u - 0x1a800000u >= 0x7f800000u - 0x1a800000u) return (double)c + (double)f;
    const float big = fmaxf(c, f), small = fminf(c, f);
    const float e = __fsub_rn(small, __fsub_rn(s, big));
    unsigned per_unit = (306u << 23) - (u & 0x7f800000u);
    if (e < 0.0f && (u & 0x007fffffu) == 0u) per_unit += 1u << 23;
    const int k = __float2int_rn(__fmul_rn(e, __uint_as_float(per_unit)));
    const long long b = ((long long)u << 29) + (896ll << 52) + (long long)k;
    return __longlong_as_double(b);
}

__device__ __forceinline__ bool between(float x, float y, float z) {
    return (y <= x && x <= z) || (y >= x && x >= z);
}

// _msm_cost, distance/_elastic.pyx:1583-1587
__device__ __forceinline__ double wave_msm_cost(float x, float y, float z, float c, double cd) {
    if (between(x, y, z)) return cd;
    const float a = fabsf(__fsub_rn(x, y));
    const float b = fabsf(__fsub_rn(x, z));
    return add_nonneg(c, b < a ? b : a);
}

__device__ __forceinline__ double abs_of(double d) { return __longlong_as_double(abs_bits(d)); }

// pair p of the job: all pairs column by column, or those above the diagonal
__device__ __forceinline__ void locate(const ElasticJob &J, int64_t p, int64_t &rs, int64_t &cs) {
    if (J.mode == PM_PAIRED) {
        rs = cs = p;
    } else if (J.mode == PM_UPPER) {
        cs = (int64_t)((1.0 + sqrt(1.0 + 8.0 * (double)p)) * 0.5);
        while (cs * (cs - 1) / 2 > p) cs--;
        while (cs * (cs + 1) / 2 <= p) cs++;
        rs = p - cs * (cs - 1) / 2;
    } else {
        cs = p / J.rows.count;
        rs = p - cs * J.rows.count;
    }
}

template <int KIND>
__global__ void __launch_bounds__(32)
    wave_pairs_kernel(const ElasticJob J, double *ring_base, int G, int64_t npairs) {
    const unsigned FULL = 0xffffffffu;
    constexpr int FR = KIND == K_MSM ? 1 : 0;
    const double INF = __longlong_as_double(0x7ff0000000000000LL);
    const int lane = threadIdx.x & 31;
    const int g = lane & (G - 1);
    const int group = lane / G, per_warp = 32 / G;
    const int64_t slots = (int64_t)gridDim.x * per_warp;
    double *ring = ring_base + (int64_t)blockIdx.x * per_warp + group;
    const int n = J.rows.len, m = J.cols.len;
    const int strips = (n - FR + kRows - 1) / kRows;
    const int rounds = (strips + G - 1) / G;
    // columns per round: lane G - 1 is done with a column before lane 0
    // fetches it in the next round, one step ahead
    const int period = imax(m, G + 2);
    const int64_t steps = (int64_t)(rounds - 1) * period + m + G - 1;
    const float cf = (float)J.c;
    const double cd = (double)cf;
    const double pen = J.penalty + J.stiffness;

    for (int64_t base = (int64_t)blockIdx.x * per_warp; base < npairs; base += slots) {
        const bool live = base + group < npairs;
        int64_t rs, cs;
        locate(J, live ? base + group : npairs - 1, rs, cs);
        const double *X = J.rows.base + rs * J.rows.stride;
        const double *Y = J.cols.base + cs * J.cols.stride;
        double gx = 0.0, gy = 0.0;
        const double *gY = nullptr;
        if constexpr (KIND == K_ERP) {
            gx = J.gsum_rows[rs];
            gy = J.gsum_cols[cs];
            gY = J.gtab_cols + cs * (int64_t)m;
        }
        double P[kRows], x[kRows];
        double rx[kRows];  // erp |x_i - g|; twe |x_{i-1} - x_i|; msm c + |x_i - x_{i-1}|
        double ad[kRows];  // twe |x_i - y| of the last column
        double st[kRows];  // twe stiffness |c - i|: a diagonal keeps its value
        float xf[kRows];
        float pxf = 0.0f;
        double xprev = 0.0;
#pragma unroll
        for (int k = 0; k < kRows; k++) P[k] = x[k] = rx[k] = ad[k] = st[k] = 0.0, xf[k] = 0.0f;
        double bot = 0.0, bdiag = 0.0, top = 0.0;
        double yp = 0.0, yn = 0.0, rn = 0.0, gn = 0.0, sn = 0.0;
        float ypf = 0.0f;
        int c = -g, strip = g;
        if (g == 0) {
            yn = __ldg(Y);
            if constexpr (KIND == K_ERP) gn = __ldg(gY);
            if constexpr (KIND == K_TWE) sn = __ldg(J.stab);
        }
        for (int64_t t = 0; t < steps; t++) {
            const double above = __shfl_up_sync(FULL, bot, 1, G);
            const bool act = c >= 0 && c < m && strip < strips;
            const double y = yn, rv = rn;
            double colv = gn;
            const double s0 = sn;
            int c1 = c + 1, s1 = strip;
            if (c1 == period) {
                c1 = 0;
                s1 += G;
            }
            if (c1 >= 0 && c1 < m && s1 < strips) {
                yn = __ldg(Y + c1);
                if constexpr (KIND == K_ERP) gn = __ldg(gY + c1);
                if constexpr (KIND == K_TWE) sn = __ldg(J.stab + abs(c1 - s1 * kRows));
                if (g == 0 && s1 > 0) rn = ring[(int64_t)c1 * slots];
            }
            if (act) {
                const float yf = (float)y;
                const int i0 = FR + strip * kRows;
                const int rows = imin(kRows, n - i0);
                if (c == 0) {
                    yp = 0.0;
#pragma unroll
                    for (int k = 0; k < kRows; k++) {
                        x[k] = k < rows ? X[i0 + k] : 0.0;
                        xf[k] = (float)x[k];
                    }
                    if constexpr (KIND != K_ERP) xprev = i0 > 0 ? X[i0 - 1] : 0.0;
                    if constexpr (KIND == K_MSM) pxf = (float)xprev;
                    if constexpr (KIND == K_ERP) bdiag = strip == 0 ? 0.0 : gx;
                    if constexpr (KIND == K_TWE) bdiag = strip == 0 ? 0.0 : INF;
#pragma unroll
                    for (int k = 0; k < kRows; k++) {
                        if constexpr (KIND == K_ERP) {
                            rx[k] = abs_of(x[k] - J.g);
                            P[k] = gx;
                        }
                        if constexpr (KIND == K_TWE) {
                            rx[k] = abs_of((k ? x[k > 0 ? k - 1 : 0] : xprev) - x[k]);
                            ad[k] = abs_of(x[k]);
                            // of the column before the first
                            st[k] = __ldg(J.stab + imin(i0 + k + 1, n - 1));
                            P[k] = INF;
                        }
                        if constexpr (KIND == K_MSM)
                            rx[k] = add_nonneg(
                                cf, fabsf(__fsub_rn(xf[k], k ? xf[k > 0 ? k - 1 : 0] : pxf)));
                    }
                }
                // the row above the strip
                double up = above;
                if (g == 0) {
                    if (strip > 0) {
                        up = rv;
                    } else if constexpr (KIND == K_MSM) {
                        // the cumulative first row; the strip's xprev is x_0
                        top = c == 0 ? abs_of(xprev - y)
                                     : top + wave_msm_cost(yf, ypf, pxf, cf, cd);
                        up = top;
                    } else {
                        up = KIND == K_ERP ? gy : INF;
                    }
                }
                const double upper = up;
                double dg = bdiag;
                if (KIND == K_MSM && c == 0) {
                    // the cumulative first column
#pragma unroll
                    for (int k = 0; k < kRows; k++) {
                        up = up + wave_msm_cost(xf[k], k ? xf[k > 0 ? k - 1 : 0] : pxf, yf, cf,
                                                cd);
                        P[k] = up;
                    }
                } else {
                    float dyf = 0.0f;
                    double adg = 0.0;
                    if constexpr (KIND == K_MSM) {
                        dyf = fabsf(__fsub_rn(yf, ypf));
                        colv = add_nonneg(cf, dyf);
                    }
                    if constexpr (KIND == K_TWE) {
                        colv = abs_of(yp - y);
                        adg = abs_of(xprev - yp);
#pragma unroll
                        for (int k = kRows - 1; k > 0; k--) st[k] = st[k - 1];
                        st[0] = s0;
                    }
                    auto column = [&](auto part) {
                        constexpr bool SHORT = decltype(part)::value;
#pragma unroll
                        for (int k = 0; k < kRows; k++) {
                            if (SHORT && k >= rows) continue;
                            const double lf = P[k];
                            double nv;
                            if constexpr (KIND == K_ERP) {
                                nv = nn_min(dg + fabs(x[k] - y), nn_min(up + rx[k], lf + colv));
                            } else if constexpr (KIND == K_MSM) {
                                const float px = k ? xf[k > 0 ? k - 1 : 0] : pxf;
                                const float fx = fabsf(__fsub_rn(xf[k], yf));
                                const float dx = fabsf(__fsub_rn(xf[k], px));
                                const double both = add_nonneg(cf, fx);
                                double cu = fx < dx ? both : rx[k];
                                if (between(xf[k], px, yf)) cu = cd;
                                double cl = dyf < fx ? colv : both;
                                if (between(yf, xf[k], ypf)) cl = cd;
                                nv = nn_min(nn_min(dg + fabs(x[k] - y), up + cu), lf + cl);
                            } else {
                                const double del = nn_min(up + rx[k], lf + colv) + pen;
                                const double a = abs_of(x[k] - y);
                                nv = nn_min(del, ((dg + a) + adg) + st[k]);
                                adg = ad[k];
                                ad[k] = a;
                            }
                            dg = lf;
                            up = nv;
                            P[k] = nv;
                        }
                    };
                    // (with one lane per pair the warp's strips have the same rows)
                    if (G == 1 && rows < kRows) column(std::true_type{});
                    else column(std::false_type{});
                }
                bot = P[kRows - 1];
                bdiag = upper;
                yp = y;
                ypf = yf;
                if (g == G - 1 && strip + 1 < strips) ring[(int64_t)c * slots] = bot;
                if (c == m - 1 && strip == strips - 1 && live) {
                    double v = P[0];
#pragma unroll
                    for (int k = 1; k < kRows; k++)
                        if (k < rows) v = P[k];
                    if (J.mode == PM_PAIRED) {
                        J.out[rs] = v;
                    } else {
                        J.out[rs * J.out_ld + cs] = v;
                        if (J.mode == PM_UPPER) J.out[cs * J.out_ld + rs] = v;
                    }
                }
            }
            c = c1;
            strip = s1;
            __syncwarp();
        }
    }
}

struct Plan {
    int lanes;
    int grid;
    int64_t pairs;
    size_t bytes;
};

// A warp that has an SM to itself takes 525 cycles for a cell of msm, one of
// many 93: their ratio.  Measured (msm, length 256, lanes 1 .. 32, ms): 9 x 10
// pairs 16.3, 8.4, 4.4, 2.4, 1.43, 0.94; 60 x 50 16.3, 8.5, 4.5, 2.6, 2.2, 2.5;
// 301 x 290 51.8, 49.4, 52.0, 50.9, 53.5, 60.8 (1 lane 48.5 since the last strip has its
// own rows only); length 60, 900 x 800: 24.7,
// 25.9, 27.1, 30.4, 60.0, 118.8.
constexpr double kAlone = 5.5;

template <int KIND>
Plan plan_kind(const ElasticJob &J) {
    Plan p;
    if (J.mode == PM_PAIRED) p.pairs = J.rows.count;
    else if (J.mode == PM_UPPER) p.pairs = J.rows.count * (J.rows.count - 1) / 2;
    else p.pairs = J.rows.count * J.cols.count;
    const int64_t sms = device_info().sm_count;
    int nb = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, wave_pairs_kernel<KIND>, 32, 0);
    const int64_t resident = (int64_t)imax(nb, 1) * sms;
    const int n = J.rows.len - (KIND == K_MSM ? 1 : 0), m = J.cols.len;
    const int64_t strips = (n + kRows - 1) / kRows;
    double best = 0.0;
    p.lanes = 0;
    if (p.pairs == 0) return Plan{1, 1, 0, 0};
    for (int G = 1; G <= 32; G *= 2) {
        const int64_t warps = (p.pairs * G + 31) / 32;
        const int64_t turns = (warps + resident - 1) / resident;
        const int64_t grid = (warps + turns - 1) / turns;
        double steps =
            (double)(((strips + G - 1) / G - 1) * (int64_t)imax(m, G + 2) + m + G - 1);
        if (G == 1) steps = (double)m * n / kRows;  // the last strip's own rows
        const double cost = (double)turns * steps *
                            std::hypot(kAlone, (double)((grid + sms - 1) / sms));
        if (!p.lanes || cost < best) {
            best = cost;
            p.lanes = G;
            p.grid = (int)std::max<int64_t>(grid, 1);
        }
    }
    p.bytes = align256((size_t)p.grid * (32 / p.lanes) * m * sizeof(double));
    return p;
}

Plan plan_wave(const ElasticJob &J) {
    switch (J.kind) {
        case K_ERP: return plan_kind<K_ERP>(J);
        case K_MSM: return plan_kind<K_MSM>(J);
        default: return plan_kind<K_TWE>(J);
    }
}

}  // namespace

// erp, msm and twe without a band edge inside the matrix, where this is the faster
// form
bool wave_supported(const ElasticJob &J) {
    if (J.kind != K_ERP && J.kind != K_MSM && J.kind != K_TWE) return false;
    if (J.key || J.all_zero || J.pending) return false;
    const char *e = getenv("WB_GPU_ELASTIC");
    if (e && (strcmp(e, "ring") == 0 || strcmp(e, "strip") == 0)) return false;
    const int n = J.rows.len, m = J.cols.len;
    const int least = J.kind == K_MSM ? 2 : 1;
    // a negative (or NaN) c has no place in add_nonneg
    if (n < least || m < least || (J.kind == K_MSM && !(J.c >= 0.0))) return false;
    if (imax(0, n - m) + J.band < n || imax(0, m - n) + J.band < m) return false;
    // Many pairs of short twe series stay with the ring kernel, whose 32 rows to a
    // column read the column's tables once: 1.03 to 1.07 times as fast (length 24 to
    // 111) where it has 6 tiles and more for each of its warps, two blocks' rings fit
    // an SM and the rows fill the tiles; with one block, or 2 to 4 tiles a warp, or
    // 100 rows (of 128), it takes 1.07 to 1.38 times as long.
    if (J.kind == K_TWE && J.mode == PM_ALL) {
        const int64_t blocks = shared_ring_blocks(J), chunks = (J.rows.count + 31) / 32;
        if (blocks >= 2 && 20 * J.rows.count >= 19 * 32 * chunks &&
            chunks * J.cols.count >= 24 * blocks * device_info().sm_count)
            return false;
    }
    return true;
}

size_t wave_bytes(const ElasticJob &J) { return plan_wave(J).bytes; }

int launch_wave(const ElasticJob &J, Workspace &ws) {
    const Plan p = plan_wave(J);
    if (p.pairs == 0) return WB_OK;
    WB_TAKE(ring, double, ws, p.bytes / sizeof(double));
    cudaStream_t s = ws.stream();
    timer_begin("wave_pairs_kernel", s);
    switch (J.kind) {
        case K_ERP: wave_pairs_kernel<K_ERP><<<p.grid, 32, 0, s>>>(J, ring, p.lanes, p.pairs); break;
        case K_MSM: wave_pairs_kernel<K_MSM><<<p.grid, 32, 0, s>>>(J, ring, p.lanes, p.pairs); break;
        default: wave_pairs_kernel<K_TWE><<<p.grid, 32, 0, s>>>(J, ring, p.lanes, p.pairs);
    }
    timer_end(s);
    WB_LAUNCH_CHECK("wave_pairs_kernel");
    return WB_OK;
}

}  // namespace wb
