// guided.cu -- FP64 dtw / wdtw / adtw distances evaluated on the cells that a
// 32-bit sweep cannot rule out, bit for bit the full FP64 recurrence.
//
// GB300 issues two FP64 operations per clock and SM, 64 times fewer than FP32,
// so a recurrence that evaluates every band cell in FP64 is bound by that pipe
// (3 operations per cell).  The value of cell (n-1, m-1), however, is the
// minimum over warping paths of a sum rounded step by step, and rounding is
// monotone: only the cells of a best path matter, and any other cell may be
// dropped (read as +inf) without changing a bit.  Per pair, one thread
//
//  1. sweeps the band in 32-bit fixed point (float32 costs rounded to units,
//     exact integer sums; strips of S rows in registers, 4 columns per step)
//     and keeps the bottom row of every strip and the cells of every S-th
//     column;
//  2. walks back from (n-1, m-1) over the S x S blocks between those kept rows
//     and columns: a block's cells are recomputed from them, every predecessor
//     whose value lies within the error bound of the cell's smallest
//     predecessor is kept as a bit, and the cells that can reach (n-1, m-1)
//     through kept predecessors are collected (bit-parallel, one word per
//     column);
//  3. runs the FP64 recurrence, with the reference's operations in its order,
//     over the collected cells (about 1.6 per row on random walks).
//
// Fixed point.  An upper bound U of the distance (a straight path through the
// band) gives a power-of-two scale of the inputs with U in (2^27, 2^29] units;
// sums saturate at kCap = 2^30, so a saturated cell costs more than the
// distance and lies on no best path.  Sums are exact; in float32 each of the
// n + m additions would add an error relative to the whole sum, which at
// length 512 keeps 1340 cells per pair instead of 835 (and 3 times as many
// steps for a warp, which waits for its widest pair).
//
// Error bound.  With d = x - y of the centred, scaled float inputs, the sum of
// a path of at most K = n + m - 1 cells differs from its exact sum on the
// float inputs by K / 2 units and a few 2^-24 of it.  The float inputs move
// the 2-norm of a path's differences by at most e sqrt(K) with
// e = 2^-24 (max|x| + max|y|).  Hence for the best predecessor p of a cell on
// a best path and any other predecessor q,
//   A(p) <= A(q) + K + 16 2^-24 A_max + 4 e sqrt(K) sqrt(A_max) + 4 e^2 K,
// A the swept values, A_max a bound of A along the path from its value at
// (n-1, m-1); the constants below are rounded up.  Predecessors outside that
// bound cannot lie on a best path.  (adtw adds a rounded penalty per move:
// K / 2 more on either side.)
//
// Pairs whose collected cells do not fit the thread's list (half of the
// band's blocks: long runs of equal values tie everywhere) or whose inputs
// are not finite are left to the full recurrence: their output holds
// kGuidedPending until launch_elastic's second pass over exactly those pairs.

#include "guided.cuh"

#include <cfloat>
#include <cstdlib>

namespace wb {

namespace {

constexpr int kThreads = 128;
constexpr unsigned kCap = 1u << 30;  // saturated value, and out of band
#define WB_GINF __int_as_float(0x7f800000)
#define WB_GINF64 __longlong_as_double(0x7ff0000000000000LL)

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

// Smallest and largest value of both series sets.
__global__ void __launch_bounds__(256)
guided_range_kernel(const SeriesSet a, const SeriesSet b, GuidedPrep *prep) {
    double lo = WB_GINF64, hi = -WB_GINF64;
    for (int set = 0; set < 2; set++) {
        const SeriesSet &S = set ? b : a;
        if (set && b.base == a.base) break;
        const int64_t total = S.count * (int64_t)S.len;
        for (int64_t t = (int64_t)blockIdx.x * 256 + threadIdx.x; t < total;
             t += (int64_t)gridDim.x * 256) {
            const int64_t s = t / S.len;
            double v = S.base[s * S.stride + (t - s * S.len)];
            if (isnan(v)) v = WB_GINF64;
            lo = v < lo ? v : lo;
            hi = v > hi ? v : hi;
        }
    }
    __shared__ long long slo[8], shi[8];
    long long l = order_code(lo), h = order_code(hi);
    for (int o = 16; o > 0; o >>= 1) {
        const long long l2 = __shfl_xor_sync(0xffffffffu, l, o);
        const long long h2 = __shfl_xor_sync(0xffffffffu, h, o);
        l = l2 < l ? l2 : l;
        h = h2 > h ? h2 : h;
    }
    if ((threadIdx.x & 31) == 0) {
        slo[threadIdx.x >> 5] = l;
        shi[threadIdx.x >> 5] = h;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; w++) {
            l = slo[w] < l ? slo[w] : l;
            h = shi[w] > h ? shi[w] : h;
        }
        atomicMin(&prep->lo, l);
        atomicMax(&prep->hi, h);
    }
}

// centre and power-of-two scale that map [lo, hi] into [-1, 1]
__device__ __forceinline__ bool centre_scale(const GuidedPrep *prep, double &centre,
                                             double &scale) {
    const double lo = order_value(prep->lo), hi = order_value(prep->hi);
    const double half = hi * 0.5 - lo * 0.5;
    if (!(isfinite(lo) && isfinite(hi) && isfinite(half))) return false;
    centre = lo * 0.5 + hi * 0.5;
    const int e = half > 0.0 ? ilogb(half) + 1 : 0;
    scale = scalbn(1.0, e < -1000 ? 1000 : -e);
    return true;
}

// Float copies of the centred, scaled series (one warp per series), padded so
// that every cell past a series' end costs +inf, and their largest magnitude.
// Row series start at element 3, which puts row 1 + S s on a 16-byte boundary.
__global__ void __launch_bounds__(256)
guided_convert_kernel(const SeriesSet rows, const SeriesSet cols, int64_t rs, int64_t cs,
                      const GuidedPrep *prep, float *xf, float *yf, float *xmax, float *ymax,
                      const double *weights, int nw, float *wext, int woff, int wlen) {
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * 256 + threadIdx.x) >> 5;
    const int64_t nwarp = ((int64_t)gridDim.x * 256) >> 5;
    double centre = 0.0, scale = 1.0;
    centre_scale(prep, centre, scale);
    for (int64_t t = warp; t < rows.count + cols.count; t += nwarp) {
        const bool row = t < rows.count;
        const int64_t s = row ? t : t - rows.count;
        const SeriesSet &S = row ? rows : cols;
        const double *src = S.base + s * S.stride;
        float *dst = row ? xf + s * rs : yf + s * cs;
        const int lead = row ? 3 : 0;
        const int total = (int)(row ? rs : cs);
        const float pad = row ? WB_GINF : -WB_GINF;
        float mx = 0.0f;
        for (int i = lane; i < total; i += 32) {
            const int e = i - lead;
            float v = pad;
            if (e >= 0 && e < S.len) {
                v = (float)((src[e] - centre) * scale);
                mx = fmaxf(mx, fabsf(v));
            }
            dst[i] = v;
        }
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        if (lane == 0) (row ? xmax : ymax)[s] = mx;
    }
    // weights by |i - j|, for i - j of either sign
    if (wext)
        for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < wlen;
             i += (int64_t)gridDim.x * 256) {
            const int d = abs((int)i - woff);
            // (a zero weight would turn an infinite cost into NaN; 1e-38 is far
            // below the bound's absolute term)
            wext[i] = fmaxf((float)weights[d < nw ? d : nw - 1], FLT_MIN);
        }
}

// --------------------------------------------------------------------------

__device__ __forceinline__ uint64_t pack2(float a, float b) {
    uint64_t p;
    asm("mov.b64 %0, {%1, %2};" : "=l"(p) : "f"(a), "f"(b));
    return p;
}

// (a - b)^2 of both halves (each rounded as the scalar operations would be)
__device__ __forceinline__ void sqdiff2(uint64_t a, uint64_t b, float &d0, float &d1) {
    asm("{\n\t.reg .b64 p;\n\tsub.rn.f32x2 p, %2, %3;\n\tmul.rn.f32x2 p, p, p;\n\t"
        "mov.b64 {%0, %1}, p;\n\t}"
        : "=f"(d0), "=f"(d1)
        : "l"(a), "l"(b));
}

// smallest predecessor (with the move's penalty) of a cell
template <int KIND>
__device__ __forceinline__ unsigned best_of(unsigned dg, unsigned up, unsigned lf, unsigned pen) {
    if constexpr (KIND == K_ADTW) return __viaddmin_u32(umin(up, lf), pen, dg);
    else return __vimin3_u32(dg, up, lf);
}

// best + cost in units, saturating (the conversion saturates at 2^31 - 1)
template <int KIND>
__device__ __forceinline__ unsigned add_cost(float sq, float w, unsigned best) {
    if constexpr (KIND == K_WDTW) sq = __fmul_rn(sq, w);
    return __viaddmin_u32(best, (unsigned)__float2int_rn(sq), kCap);
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
    __device__ __forceinline__ Band(const GuidedArgs &A, int S)
        : n(A.J.rows.len), m(A.J.cols.len), r(A.J.band), mx(imax(0, m - n) + r),
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

// One column of a strip: Pin holds column c - 1, Pout receives column c;
// wq[S - 1 - k] is the weight of row k.
template <int KIND, int S, bool MASK>
__device__ __forceinline__ void sweep_column(const unsigned (&Pin)[S], unsigned (&Pout)[S],
                                             unsigned bup, unsigned bdiag,
                                             const uint64_t (&x2)[S / 2], float y,
                                             const float *wq, unsigned pen, unsigned M) {
    const uint64_t yy = pack2(y, y);
#pragma unroll
    for (int k = 0; k < S; k += 2) {
        float sq[2];
        sqdiff2(x2[k / 2], yy, sq[0], sq[1]);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int i = k + h;
            const unsigned dg = i == 0 ? bdiag : Pin[i > 0 ? i - 1 : 0];
            const unsigned up = i == 0 ? bup : Pout[i > 0 ? i - 1 : 0];
            const float w = KIND == K_WDTW ? wq[S - 1 - i] : 1.0f;
            unsigned v = add_cost<KIND>(sq[h], w, best_of<KIND>(dg, up, Pin[i], pen));
            if (MASK) v = ((M >> i) & 1u) ? v : kCap;
            Pout[i] = v;
        }
    }
}

// An upper bound of the distance's sum: the path through the cells nearest to
// the straight line from (0, 0) to (n-1, m-1), one per row (or per column, the
// longer of the two), which the band always holds.
template <int KIND>
__device__ __forceinline__ float straight_path(const GuidedArgs &A, const Band &B,
                                               const float *__restrict__ xr,
                                               const float *__restrict__ yr, float pen) {
    const int steps = imax(B.n, B.m), other = imin(B.n, B.m);
    float sum = 0.0f;
    int at = 0, rem = 0;  // at = floor(i (other - 1) / (steps - 1))
#pragma unroll 4
    for (int i = 0; i < steps; i++) {
        const int r = B.n >= B.m ? i : at, c = B.n >= B.m ? at : i;
        const float d = __fsub_rn(xr[3 + r], yr[c]);
        float sq = __fmul_ru(d, d);
        // (row 0 weighs column c with index c - 1)
        if constexpr (KIND == K_WDTW)
            sq = __fmul_ru(sq, fmaxf(A.wext[A.woff + c - r], A.wext[A.woff + imax(c - r - 1, 0)]));
        sum = __fadd_ru(sum, sq);
        rem += other - 1;
        const bool step = rem >= steps - 1;
        if (step) {
            rem -= steps - 1;
            at++;
        }
        if (KIND == K_ADTW && !step) sum = __fadd_ru(sum, pen);
    }
    // the differences' roundings
    return __fmul_ru(sum, 1.000001f);
}

// Step 1: the sweep; returns the value of cell (n-1, m-1) in units.  xr, yr:
// the pair's padded float series, su: their scale; all lanes of a warp share
// the band.
template <int KIND, int S>
__device__ __forceinline__ unsigned guided_sweep(const GuidedArgs &A, const Band &B,
                                                 const float *__restrict__ xr,
                                                 const float *__restrict__ yr, int64_t gt,
                                                 float su, unsigned pen) {
    constexpr int LG = S == 8 ? 1 : 2;  // groups of 4 columns per block, as a shift
    const int64_t nth = A.nth;
    const int G = A.groups, NB = A.blocks;
    const uint4 CAP4 = make_uint4(kCap, kCap, kCap, kCap);
    const float4 *y4 = reinterpret_cast<const float4 *>(yr);
    unsigned result = kCap;
    // row 0: cumulative, without penalties, weight index j - 1
    {
        const float x0 = __fmul_rn(xr[3], su);
        const int lim = imin(B.m, B.mx);
        unsigned acc = 0;
        for (int g = 0; g <= (lim - 1) >> 2; g++) {
            const float4 y = y4[g];
            const float yq[4] = {y.x, y.y, y.z, y.w};
            unsigned v[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int c = 4 * g + q;
                const float d = __fsub_rn(x0, __fmul_rn(yq[q], su));
                const float w = KIND == K_WDTW ? A.wext[A.woff + imax(c - 1, 0)] : 1.0f;
                acc = add_cost<KIND>(__fmul_rn(d, d), w, acc);
                v[q] = c < lim ? acc : kCap;
            }
            A.ckrow[(int64_t)g * nth + gt] = make_uint4(v[0], v[1], v[2], v[3]);
        }
    }
    int pg0 = 0, pg1 = (B.ce(-1, S) - 1) >> 2;
    for (int s = 0; s < B.ns; s++) {
        const int i0 = 1 + s * S;
        const int rows = imin(S, B.n - i0);
        const int cs = B.cs(s, S), ce = B.ce(s, S);
        const int g0 = cs >> 2, g1 = (ce - 1) >> 2;
        // columns where every row of the strip is in band, the last column
        // of the last strip excepted (it yields the result)
        int bstart = 0x7fffffff, bend = 0;
        if (rows == S) {
            bstart = imax(cs, i0 + S - 1 + B.lo);
            bend = imin(s == B.ns - 1 ? imin(ce, (B.m - 1) & ~3) : ce, i0 + B.mx);
        }
        uint64_t x2[S / 2];
        const float4 *x4 = reinterpret_cast<const float4 *>(xr + 3 + i0);
#pragma unroll
        for (int k = 0; k < S / 4; k++) {
            const float4 t = x4[k];
            x2[2 * k] = pack2(__fmul_rn(t.x, su), __fmul_rn(t.y, su));
            x2[2 * k + 1] = pack2(__fmul_rn(t.z, su), __fmul_rn(t.w, su));
        }
        const uint4 *in = A.ckrow + ((int64_t)s * G - pg0) * nth + gt;
        uint4 *out = A.ckrow + ((int64_t)(s + 1) * G - g0) * nth + gt;
        uint4 *col = A.ckcol + ((int64_t)s * NB - (g0 >> LG)) * (S / 4) * nth + gt;
        auto up4 = [&](int g) { return g >= pg0 && g <= pg1 ? in[(int64_t)g * nth] : CAP4; };
        unsigned P[S], Q[S];
#pragma unroll
        for (int k = 0; k < S; k++) P[k] = kCap;
        unsigned bd = up4(g0 - 1).w;
        uint4 nu = up4(g0);
        float4 ny = y4[g0];
        for (int g = g0; g <= g1; g++) {
            const uint4 u = nu;
            const float4 y = make_float4(__fmul_rn(ny.x, su), __fmul_rn(ny.y, su),
                                         __fmul_rn(ny.z, su), __fmul_rn(ny.w, su));
            if (g < g1) {
                nu = up4(g + 1);
                ny = y4[g + 1];
            }
            float w[S + 4];
            if constexpr (KIND == K_WDTW) {
                const float4 *w4 = reinterpret_cast<const float4 *>(
                    A.wext + (A.woff + 4 * g - i0 - (S - 1)));
#pragma unroll
                for (int k = 0; k < S / 4 + 1; k++) {
                    const float4 t = w4[k];
                    w[4 * k] = t.x;
                    w[4 * k + 1] = t.y;
                    w[4 * k + 2] = t.z;
                    w[4 * k + 3] = t.w;
                }
            }
            uint4 o;
            if (4 * g >= bstart && 4 * g + 3 < bend) {
                sweep_column<KIND, S, false>(P, Q, u.x, bd, x2, y.x, w, pen, 0u);
                o.x = Q[S - 1];
                sweep_column<KIND, S, false>(Q, P, u.y, u.x, x2, y.y, w + 1, pen, 0u);
                o.y = P[S - 1];
                sweep_column<KIND, S, false>(P, Q, u.z, u.y, x2, y.z, w + 2, pen, 0u);
                o.z = Q[S - 1];
                sweep_column<KIND, S, false>(Q, P, u.w, u.z, x2, y.w, w + 3, pen, 0u);
                o.w = P[S - 1];
            } else {
                const int e = 4 * g - i0 - B.lo;
                auto masked = [&](int q, const unsigned(&Pin)[S], unsigned(&Pout)[S],
                                  unsigned bup, unsigned bdg, float yq) {
                    const unsigned M = band_rows(e + q, B.width);
                    sweep_column<KIND, S, true>(Pin, Pout, bup, bdg, x2, yq, w + q, pen, M);
                    if (s == B.ns - 1 && 4 * g + q == B.m - 1) {
#pragma unroll
                        for (int k = 0; k < S; k++)
                            if (k < rows) result = Pout[k];
                    }
                };
                masked(0, P, Q, u.x, bd, y.x);
                o.x = Q[S - 1];
                masked(1, Q, P, u.y, u.x, y.y);
                o.y = P[S - 1];
                masked(2, P, Q, u.z, u.y, y.z);
                o.z = Q[S - 1];
                masked(3, Q, P, u.w, u.z, y.w);
                o.w = P[S - 1];
            }
            bd = u.w;
            out[(int64_t)g * nth] = o;
            if (((g + 1) & ((1 << LG) - 1)) == 0) {
                uint4 *cd = col + (int64_t)(g >> LG) * (S / 4) * nth;
#pragma unroll
                for (int k = 0; k < S / 4; k++)
                    cd[k * nth] = make_uint4(P[4 * k], P[4 * k + 1], P[4 * k + 2],
                                             P[4 * k + 3]);
            }
        }
        pg0 = g0;
        pg1 = g1;
    }
    return result;
}

// shift the sign bit of `v` into `bits`
__device__ __forceinline__ unsigned push_sign(unsigned bits, int v) {
    return __funnelshift_l((unsigned)v, bits, 1);
}

// Step 2 of one block: cells (i0 + k, c0 + q), k, q < S, from the kept row
// above, the kept column left of it, with the excluded-predecessor bits of
// every column (row 0 of the block in the highest of the S bits).
template <int KIND, int S>
__device__ __forceinline__ void block_bits(const GuidedArgs &A, const Band &B, int s, int b,
                                           const float *__restrict__ xr,
                                           const float *__restrict__ yr, int64_t gt, float su,
                                           unsigned pen, unsigned tol, unsigned (&xd)[S],
                                           unsigned (&xu)[S], unsigned (&xl)[S]) {
    constexpr int LG = S == 8 ? 1 : 2;
    const int64_t nth = A.nth;
    const int i0 = 1 + s * S, c0 = b * S;
    uint64_t x2[S / 2];
    const float4 *x4 = reinterpret_cast<const float4 *>(xr + 3 + i0);
    const float4 *y4 = reinterpret_cast<const float4 *>(yr + c0);
    unsigned P[S], Q[S], top[S];
    float yv[S], w[2 * S];
#pragma unroll
    for (int k = 0; k < S / 4; k++) {
        const float4 t = x4[k], u = y4[k];
        x2[2 * k] = pack2(__fmul_rn(t.x, su), __fmul_rn(t.y, su));
        x2[2 * k + 1] = pack2(__fmul_rn(t.z, su), __fmul_rn(t.w, su));
        yv[4 * k] = __fmul_rn(u.x, su);
        yv[4 * k + 1] = __fmul_rn(u.y, su);
        yv[4 * k + 2] = __fmul_rn(u.z, su);
        yv[4 * k + 3] = __fmul_rn(u.w, su);
    }
    // row i0 - 1, from the strip above (the row-0 slot for s = 0)
    const int pg0 = B.cs(s - 1, S) >> 2, pg1 = (B.ce(s - 1, S) - 1) >> 2;
    const uint4 *in = A.ckrow + ((int64_t)s * A.groups - pg0) * nth + gt;
    const int gb = c0 >> 2;
#pragma unroll
    for (int k = 0; k < S / 4; k++) {
        const int g = gb + k;
        uint4 t = make_uint4(kCap, kCap, kCap, kCap);
        if (g >= pg0 && g <= pg1) t = in[(int64_t)g * nth];
        top[4 * k] = t.x;
        top[4 * k + 1] = t.y;
        top[4 * k + 2] = t.z;
        top[4 * k + 3] = t.w;
    }
    unsigned bd = kCap;
    if (gb - 1 >= pg0 && gb - 1 <= pg1) bd = in[(int64_t)(gb - 1) * nth].w;
    // column c0 - 1 of this strip
    const int g0 = B.cs(s, S) >> 2;
    const bool have = gb - 1 >= g0;
    const uint4 *col =
        A.ckcol + ((int64_t)s * A.blocks + (b - 1) - (g0 >> LG)) * (S / 4) * nth + gt;
#pragma unroll
    for (int k = 0; k < S / 4; k++) {
        uint4 t = make_uint4(kCap, kCap, kCap, kCap);
        if (have) t = col[k * nth];
        P[4 * k] = t.x;
        P[4 * k + 1] = t.y;
        P[4 * k + 2] = t.z;
        P[4 * k + 3] = t.w;
    }
    if constexpr (KIND == K_WDTW) {
        const float4 *w4 =
            reinterpret_cast<const float4 *>(A.wext + (A.woff + c0 - i0 - (S - 1)));
#pragma unroll
        for (int k = 0; k < S / 2; k++) {
            const float4 t = w4[k];
            w[4 * k] = t.x;
            w[4 * k + 1] = t.y;
            w[4 * k + 2] = t.z;
            w[4 * k + 3] = t.w;
        }
    }
    // cells outside the band by their diagonal q - k
    unsigned out_of_band[2 * S - 1];
#pragma unroll
    for (int t = 0; t < 2 * S - 1; t++) {
        const int e = c0 - i0 + (t - (S - 1)) - B.lo;
        out_of_band[t] = (unsigned)e < (unsigned)B.width ? 0u : kCap;
    }
#pragma unroll
    for (int q = 0; q < S; q++) {
        const uint64_t yy = pack2(yv[q], yv[q]);
        unsigned bd_ = 0, bu_ = 0, bl_ = 0;
#pragma unroll
        for (int k = 0; k < S; k += 2) {
            float sq[2];
            sqdiff2(x2[k / 2], yy, sq[0], sq[1]);
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int i = k + h, j = i > 0 ? i - 1 : 0;
                const unsigned dg = i == 0 ? (q == 0 ? bd : top[q > 0 ? q - 1 : 0]) : P[j];
                const unsigned up = i == 0 ? top[q] : Q[j];
                const unsigned lf = P[i];
                const unsigned best = best_of<KIND>(dg, up, lf, pen);
                const int t = (int)(best + tol);
                const int tm = KIND == K_ADTW ? t - (int)pen : t;
                bd_ = push_sign(bd_, t - (int)dg);
                bu_ = push_sign(bu_, tm - (int)up);
                bl_ = push_sign(bl_, tm - (int)lf);
                const unsigned v =
                    add_cost<KIND>(sq[h], KIND == K_WDTW ? w[q - i + S - 1] : 1.0f, best);
                Q[i] = umax(v, out_of_band[q - i + S - 1]);
            }
        }
        xd[q] = bd_;
        xu[q] = bu_;
        xl[q] = bl_;
#pragma unroll
        for (int k = 0; k < S; k++) P[k] = Q[k];
    }
}

// Cells of one column reachable upwards from `r` through cells whose up move
// is not excluded; bit S of the result: the move out of the block's top row.
template <int S>
__device__ __forceinline__ unsigned fill_up(unsigned r, unsigned xu) {
    const unsigned up = ~xu & ((1u << S) - 1u);
    unsigned p = up;
    r |= (r & p) << 1;
    p &= p >> 1;
    r |= (r & p) << 2;
    p &= p >> 2;
    r |= (r & p) << 4;
    if (S > 8) {
        p &= p >> 4;
        r |= (r & p) << 8;
    }
    // the steps add up to S - 1 rows; a run through the whole column is S
    return r | ((r & up) << 1);
}

template <int KIND, int S>
__global__ void __launch_bounds__(kThreads, S == 8 ? 4 : 3)
guided_pairs_kernel(const GuidedArgs A) {
    constexpr int W64 = S * S / 64;     // mask words of a block
    constexpr int EW = 2 * W64 + 1;     // list words of a block: position, mask
    constexpr unsigned SM = (1u << S) - 1u;
    __shared__ double vs[S][kThreads];  // last FP64 value of every block row
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int64_t nth = A.nth;
    const int64_t gt = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    const ElasticJob &J = A.J;
    const Band B(A, S);
    const double INF = WB_GINF64;
    double centre = 0.0, scale = 1.0;
    const bool finite = centre_scale(A.prep, centre, scale);
    const float penf = KIND == K_ADTW ? __double2float_ru(J.p * scale * scale) : 0.0f;
    const int64_t chunks = (J.rows.count + 31) >> 5;
    const int64_t ntiles = J.mode == PM_PAIRED ? chunks : chunks * J.cols.count;
    const float K = (float)(B.n + B.m);

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
        bool active = rs < J.rows.count && !(J.mode == PM_UPPER && rs >= cs);
        if (!__any_sync(FULL, active)) continue;
        if (!active) {  // sweeps along on a valid pair
            rs = J.rows.count - 1;
            cs = J.mode == PM_PAIRED ? rs : cs;
        }
        const float *xr = A.xf + rs * A.xs;
        const float *yr = A.yf + cs * A.ys;
        // the power of two that brings the upper bound into (2^27, 2^29] units
        const float ub = fmaxf(straight_path<KIND>(A, B, xr, yr, penf), 1e-30f);
        bool live = active && finite && ub < 1e30f;
        const int half = (29 - ilogbf(ub) - 1) >> 1;
        const float su = live ? scalbnf(1.0f, half) : 1.0f;
        const unsigned pen =
            KIND == K_ADTW ? (unsigned)__float2int_rn(fminf(__fmul_rn(__fmul_rn(penf, su), su),
                                                            (float)kCap))
                           : 0u;
        const unsigned au = guided_sweep<KIND, S>(A, B, xr, yr, gt, su, pen);

        // the bound (file header) in units; sqrt(A_max) <= sqrt(A + K) (1 + 2^-22) + 2 e sqrt(K)
        const float e = __fmul_ru(su, __fmaf_ru(6.0e-8f, __fadd_ru(A.xmax[rs], A.ymax[cs]), 1e-37f));
        const float ek = __fmul_ru(e, __fsqrt_ru(K));
        const float ra = __fmaf_ru(2.1f, ek, __fmul_ru(__fsqrt_ru(__fadd_ru((float)au, K)), 1.000001f));
        const float tolf = __fadd_ru(
            __fmaf_ru(KIND == K_ADTW ? 2.02f : 1.01f, K, __fmul_ru(1.2e-6f, __fmul_ru(ra, ra))),
            __fadd_ru(__fmul_ru(__fmul_ru(4.2f, ek), __fadd_ru(ra, ek)), 8.0f));
        live = live && au < kCap && tolf < 2.5e8f;
        const unsigned tol = live ? (unsigned)tolf : 0u;
        const bool swept = live;

        // ---- step 2: collect cells, from the last strip up
        int s = B.ns - 1, b = (B.m - 1) / S;
        int slo = B.m - 1, shi = B.m - 1;       // seeds in the strip's bottom row
        int nlo = 0x7fffffff, nhi = -1;         // seeds of the strip above
        unsigned carry = 0;                     // cells reached in the column left of the block
        int idx = 0;
        while (__any_sync(FULL, live)) {
            if (live) {
                unsigned xd[S], xu[S], xl[S];
                block_bits<KIND, S>(A, B, s, b, xr, yr, gt, su, pen, tol, xd, xu, xl);
                const int c0 = b * S;
                const int rows = imin(S, B.n - 1 - s * S);
                const unsigned bottom = 1u << (S - rows);
                uint64_t mask[W64];
#pragma unroll
                for (int w = 0; w < W64; w++) mask[w] = 0;
                unsigned from = carry;
#pragma unroll
                for (int q = S - 1; q >= 0; q--) {
                    const int c = c0 + q;
                    unsigned r = from;
                    if (c >= slo && c <= shi) r |= bottom;
                    r = fill_up<S>(r, xu[q]);
                    const unsigned dg = (r & SM & ~xd[q]) << 1;
                    if (r >> S) {
                        nlo = imin(nlo, c);
                        nhi = imax(nhi, c);
                    }
                    if (dg >> S) {
                        nlo = imin(nlo, c - 1);
                        nhi = imax(nhi, c - 1);
                    }
                    r &= SM;
                    from = ((r & ~xl[q]) | dg) & SM;
                    mask[q * S / 64] |= (uint64_t)r << (64 - S - (q * S) % 64);
                }
                carry = from;
                uint32_t *ent = A.list + (int64_t)idx * EW * nth + gt;
                ent[0] = ((uint32_t)s << 16) | (uint32_t)b;
#pragma unroll
                for (int w = 0; w < W64; w++) {
                    ent[(1 + 2 * w) * nth] = (uint32_t)(mask[w] >> 32);
                    ent[(2 + 2 * w) * nth] = (uint32_t)mask[w];
                }
                idx++;
                if (carry != 0 || slo < c0) {
                    b--;
                } else {
                    slo = nlo;
                    shi = nhi;
                    nlo = 0x7fffffff;
                    nhi = -1;
                    b = shi / S;
                    s--;
                    if (s < 0) {
                        live = false;
                        if (shi < 0) idx = -1;
                    }
                }
                if (live && (idx == A.list_cap || b < 0 || shi < 0)) {
                    live = false;
                    idx = -1;  // the list is full
                }
            }
        }
        const bool ok = swept && idx > 0;

        // ---- step 3: FP64 over the collected cells, in order
        double value = 0.0;
        if (__any_sync(FULL, ok)) {
            const double *X = J.rows.base + rs * J.rows.stride;
            const double *Y = J.cols.base + cs * J.cols.stride;
            double *brow = A.brow + gt;
            const int64_t mp = A.brow_cols;
            const int hi0 = ok ? shi : -1;
            if (ok) {
                const double x0 = X[0];
                double acc = 0.0;
                for (int c = 0; c <= hi0; c++) {
                    const double v = x0 - __ldg(Y + c);
                    double cst = v * v;
                    if (KIND == K_WDTW) cst = cst * __ldg(J.weights + imax(c - 1, 0));
                    acc = c == 0 ? cst : acc + cst;
                    brow[c * nth] = acc;
                }
            }
            int plo = 0, phi = -1, clo = 0, chi = hi0;  // columns held by brow
            int cur = -1;
            unsigned lm = 0;  // collected rows of the column left of the block
            int ei = ok ? idx - 1 : -1;
            while (__any_sync(FULL, ei >= 0)) {
                if (ei >= 0) {
                    const uint32_t *ent = A.list + (int64_t)ei * EW * nth + gt;
                    const uint32_t h = ent[0];
                    const int bs = (int)(h >> 16), bb = (int)(h & 0xffffu);
                    if (bs != cur) {
                        plo = clo;
                        phi = chi;
                        clo = bb * S;
                        lm = 0;
                        cur = bs;
                    }
                    chi = bb * S + S - 1;
                    const double *above = brow + (int64_t)(bs & 1) * mp * nth;
                    double *below = brow + (int64_t)((bs + 1) & 1) * mp * nth;
                    const int i0 = 1 + bs * S;
#pragma unroll 1
                    for (int w = 0; w < W64; w++) {
                        const uint64_t M = ((uint64_t)ent[(1 + 2 * w) * nth] << 32) |
                                           ent[(2 + 2 * w) * nth];
                        const uint64_t LM = (M >> S) | ((uint64_t)lm << (64 - S));
                        const int cw = bb * S + w * (64 / S);
#pragma unroll
                        for (int q = 0; q < 64 / S; q++)
                            if (!((M >> (64 - S - q * S)) & 1u)) below[(int64_t)(cw + q) * nth] = INF;
                        uint64_t todo = M;
                        double last = 0.0, last_old = 0.0;
                        while (todo) {
                            const int p = __clzll((long long)todo);
                            const uint64_t bit = 0x8000000000000000ULL >> p;
                            todo ^= bit;
                            const int k = p & (S - 1);
                            const int c = cw + p / S;
                            const double d = X[i0 + k] - __ldg(Y + c);
                            double cst = d * d;
                            if (KIND == K_WDTW) cst = cst * __ldg(J.weights + abs(i0 + k - c));
                            const double old = vs[k][threadIdx.x];
                            const double lf = (LM & bit) ? old : INF;
                            double up, dg;
                            if (k > 0) {
                                const bool hu = (M & (bit << 1)) != 0;
                                up = hu ? last : INF;
                                dg = INF;
                                if (LM & (bit << 1)) dg = hu ? last_old : vs[k - 1][threadIdx.x];
                            } else {
                                up = c >= plo && c <= phi ? above[(int64_t)c * nth] : INF;
                                dg = c - 1 >= plo && c - 1 <= phi ? above[(int64_t)(c - 1) * nth]
                                                                  : INF;
                            }
                            double mv = nn_min(up, lf);
                            if (KIND == K_ADTW) mv = mv + J.p;
                            const double nv = nn_min(mv, dg) + cst;
                            vs[k][threadIdx.x] = nv;
                            last = nv;
                            last_old = old;
                            if (k == S - 1) below[(int64_t)c * nth] = nv;
                            value = nv;
                        }
                        lm = (unsigned)(M & SM);
                    }
                    ei--;
                }
            }
        }
        if (active) {
            const double res = ok ? sqrt(value) : __longlong_as_double(kGuidedPending);
            if (J.mode == PM_PAIRED) {
                J.out[rs] = res;
            } else {
                J.out[rs * J.out_ld + cs] = res;
                if (J.mode == PM_UPPER) J.out[cs * J.out_ld + rs] = res;
            }
            if (!ok) atomicAdd(&A.prep->pending, 1ull);
        }
    }
}

// --------------------------------------------------------------------------
// host side

struct Plan {
    bool use = false;
    int S = 8, grid = 0;
    int groups = 0, blocks = 0, list_cap = 0, brow_cols = 0;
    int64_t xs = 0, ys = 0;
    int woff = 0, wlen = 0;
    size_t shared_bytes = 0;  // float copies, magnitudes, weights, prep
    size_t thread_bytes = 0;  // per resident thread
};

template <int KIND>
int blocks_per_sm(int S) {
    int nb = 0;
    if (S == 8)
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, guided_pairs_kernel<KIND, 8>, kThreads, 0);
    else
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, guided_pairs_kernel<KIND, 16>, kThreads, 0);
    return nb;
}

int64_t round_up(int64_t v, int64_t a) { return (v + a - 1) / a * a; }

// per-thread memory budget of the kept rows and columns of all resident pairs
constexpr size_t kGuidedBudget = (size_t)8 << 30;

Plan plan_guided(const ElasticJob &J, size_t avail) {
    Plan p;
    const int n = J.rows.len, m = J.cols.len, r = J.band;
    if (J.kind != K_DTW && J.kind != K_WDTW && J.kind != K_ADTW) return p;
    if (J.key || J.all_zero || J.pending) return p;
    const char *e = getenv("WB_GPU_ELASTIC");
    if (e && (strcmp(e, "ring") == 0 || strcmp(e, "strip") == 0)) return p;
    const int mx = imax(0, m - n) + r, mn = imax(0, n - m);
    const int width = mx + mn + r - 1;
    if (imin(n, m) < 24 || imin(width, m) < 12) return p;
    if ((int64_t)n + m > 1 << 15) return p;  // positions are 16 bits
    const DeviceInfo &dev = device_info();
    const int64_t work = (J.mode == PM_PAIRED ? (J.rows.count + 31) / 32
                                              : (J.rows.count + 31) / 32 * J.cols.count) * 32;
    const int64_t want = (work + kThreads - 1) / kThreads;
    for (int S = 8; S <= 16; S += 8) {
        const int ns = (n - 1 + S - 1) / S;
        p.S = S;
        p.groups = (imin(m, width + S - 1) + 3) / 4 + 1;
        p.blocks = p.groups / (S / 4) + 2;
        p.list_cap = imax((n + m) / S + 8, ns * p.blocks / 2);
        p.brow_cols = (int)round_up(m, S);
        p.xs = round_up(3 + 1 + (int64_t)ns * S, 4);
        p.ys = round_up(m, 16);
        p.woff = (int)round_up(n + 2 * S, 4);
        p.wlen = J.kind == K_WDTW ? (int)round_up(p.woff + m + 2 * S, 4) : 0;
        const int EW = S * S / 32 + 1;
        p.thread_bytes = (size_t)(ns + 1) * p.groups * 16 + (size_t)ns * p.blocks * S * 4 +
                         (size_t)p.list_cap * EW * 4 + (size_t)2 * p.brow_cols * 8;
        p.shared_bytes = align256(J.rows.count * p.xs * 4) + align256(J.cols.count * p.ys * 4) +
                         align256(J.rows.count * 4) + align256(J.cols.count * 4) +
                         align256((size_t)imax(p.wlen, 1) * 4) + align256(sizeof(GuidedPrep)) +
                         4 * 256;
        int nb;
        switch (J.kind) {
            case K_DTW: nb = blocks_per_sm<K_DTW>(S); break;
            case K_WDTW: nb = blocks_per_sm<K_WDTW>(S); break;
            default: nb = blocks_per_sm<K_ADTW>(S); break;
        }
        const int64_t full = std::min<int64_t>(want, (int64_t)imax(nb, 1) * dev.sm_count);
        size_t room = std::min(kGuidedBudget, avail > p.shared_bytes ? avail - p.shared_bytes : 0);
        const int64_t fit = (int64_t)(room / (p.thread_bytes * kThreads));
        p.grid = (int)std::min(full, fit);
        // enough resident pairs to keep the SMs busy, else larger blocks or
        // the full recurrence
        const int64_t enough = S == 8 ? full : std::min<int64_t>(full, dev.sm_count);
        p.use = p.grid >= 1 && p.grid >= enough;
        if (p.use) return p;
    }
    return p;
}

template <int KIND>
int run_kernel(const GuidedArgs &A, int S, int grid, cudaStream_t s) {
    timer_begin("guided_pairs_kernel", s);
    if (S == 8) guided_pairs_kernel<KIND, 8><<<grid, kThreads, 0, s>>>(A);
    else guided_pairs_kernel<KIND, 16><<<grid, kThreads, 0, s>>>(A);
    timer_end(s);
    WB_LAUNCH_CHECK("guided_pairs_kernel");
    return WB_OK;
}

}  // namespace

size_t guided_workspace_bytes(const ElasticJob &J) {
    const Plan p = plan_guided(J, SIZE_MAX);
    if (!p.use) return 0;
    return p.shared_bytes + 2 * 4096 + p.thread_bytes * (size_t)p.grid * kThreads;
}

int launch_guided(const ElasticJob &J, Workspace &ws, size_t leave,
                  unsigned long long **pending) {
    *pending = nullptr;
    leave += 4096;  // and the alignment of the pieces
    const size_t avail = ws.remaining();
    const Plan p = plan_guided(J, avail > leave ? avail - leave : 0);
    if (!p.use) return WB_OK;
    cudaStream_t s = ws.stream();
    const int ns = (J.rows.len - 1 + p.S - 1) / p.S;
    const int64_t nth = (int64_t)p.grid * kThreads;
    GuidedArgs A;
    A.J = J;
    A.nth = nth;
    A.groups = p.groups;
    A.blocks = p.blocks;
    A.list_cap = p.list_cap;
    A.brow_cols = p.brow_cols;
    A.xs = p.xs;
    A.ys = p.ys;
    A.woff = p.woff;
    WB_TAKE(prep, GuidedPrep, ws, 1);
    WB_TAKE(xf, float, ws, J.rows.count * p.xs);
    WB_TAKE(yf, float, ws, J.cols.count * p.ys);
    WB_TAKE(xmax, float, ws, J.rows.count);
    WB_TAKE(ymax, float, ws, J.cols.count);
    WB_TAKE(wext, float, ws, imax(p.wlen, 1));
    WB_TAKE(ckrow, uint4, ws, (size_t)(ns + 1) * p.groups * nth);
    WB_TAKE(ckcol, uint4, ws, (size_t)ns * p.blocks * (p.S / 4) * nth);
    WB_TAKE(list, uint32_t, ws, (size_t)p.list_cap * (p.S * p.S / 32 + 1) * nth);
    WB_TAKE(brow, double, ws, (size_t)2 * p.brow_cols * nth);
    A.prep = prep;
    A.xf = xf;
    A.yf = yf;
    A.xmax = xmax;
    A.ymax = ymax;
    A.wext = wext;
    A.ckrow = ckrow;
    A.ckcol = ckcol;
    A.list = list;
    A.brow = brow;
    // lo = the largest code, hi = the smallest, the counters zero
    WB_CUDA(cudaMemsetAsync(&prep->lo, 0x7f, sizeof(prep->lo), s));
    WB_CUDA(cudaMemsetAsync(&prep->hi, 0x80, sizeof(prep->hi), s));
    WB_CUDA(cudaMemsetAsync(&prep->queue, 0, 2 * sizeof(prep->queue), s));
    const int64_t cap = (int64_t)device_info().sm_count * 4;
    const int64_t values = J.rows.count * J.rows.len + J.cols.count * J.cols.len;
    guided_range_kernel<<<(int)std::min(cap, (values + 1023) / 1024), 256, 0, s>>>(
        J.rows, J.cols, prep);
    WB_LAUNCH_CHECK("guided_range_kernel");
    const int64_t series = J.rows.count + J.cols.count;
    const int nw = J.kind == K_WDTW ? imax(J.rows.len, J.cols.len) : 0;
    guided_convert_kernel<<<(int)std::min(cap, (series + 7) / 8), 256, 0, s>>>(
        J.rows, J.cols, p.xs, p.ys, prep, xf, yf, xmax, ymax, J.weights, nw,
        p.wlen ? wext : nullptr, p.woff, p.wlen);
    WB_LAUNCH_CHECK("guided_convert_kernel");
    switch (J.kind) {
        case K_DTW: WB_TRY(run_kernel<K_DTW>(A, p.S, p.grid, s)); break;
        case K_WDTW: WB_TRY(run_kernel<K_WDTW>(A, p.S, p.grid, s)); break;
        default: WB_TRY(run_kernel<K_ADTW>(A, p.S, p.grid, s)); break;
    }
    *pending = &prep->pending;
    return WB_OK;
}

}  // namespace wb
