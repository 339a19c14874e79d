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
//  1. sweeps the band in 32-bit fixed point (exact integer sums; strips of S
//     rows in registers, 4 columns per step) and keeps the bottom row of every
//     strip and the cells of every S-th column (one byte per cell for S = 8,
//     which the DRAM writes bound at about 8 ms for the shape below; S = 16
//     halves it where S = 8 would not fit its budget);
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
// steps for a warp, which waits for its widest pair).  A cost is the high half
// of the square of a 31-bit difference (three instructions per cell: subtract,
// 3-input minimum, multiply-add); where the largest difference of a pair is
// far above its distance, and for wdtw, the warp takes float32 costs rounded to
// units instead (the conversion issues at 16 per clock and SM and takes most
// of that sweep's time, which hides the low parts of the inputs: without them
// the inputs' rounding, unweighted, kept 467 instead of 155 blocks per pair for
// wdtw at length 569, 17.3 instead of 6.3 ms for 143 x 6 pairs).
//
// Error bound.  With d = x - y of the centred, scaled, rounded inputs, the sum
// of a path of at most K = n + m - 1 cells differs from its exact sum on these
// inputs by K / 2 units and a few 2^-24 of it (float costs) or lies at most K
// units below it (fixed point).  Rounding the inputs moves the 2-norm of a
// path's differences by at most e sqrt(K), e = 2^-47 (max|x| + max|y|) for
// float inputs with their low parts and two roundings of the shifted values for
// fixed-point ones.  Hence for the best predecessor p of a cell on
// a best path and any other predecessor q,
//   A(p) <= A(q) + K + 16 2^-24 A_max + 4 e sqrt(K) sqrt(A_max) + 4 e^2 K,
// A the swept values, A_max a bound of A along the path from its value at
// (n-1, m-1); the constants below are rounded up.  Predecessors outside that
// bound cannot lie on a best path, nor can saturated ones: the sums along the
// path stay below A_max, and pairs whose bound would reach from there to kCap are
// not taken.  (adtw adds a rounded penalty per move: K / 2 more on either side,
// and in fixed point too 2^-23 + 2^-24 of A_max on either side, since the penalty
// is a float before it is in units.)
//
// Pairs whose collected cells do not fit the thread's list (a fourth of the band's
// blocks, half of a narrow band's: long runs of equal values tie everywhere) or whose
// inputs are not finite are left to the full recurrence: their output holds
// kGuidedPending, and a list of them goes to guided_tail_kernel (few pairs) or to
// launch_elastic's second pass.
//
// Measured on one GB300 (full recurrence -> guided): dtw r = 0.1, 1000 x 1000,
// length 512: 292 -> 36 ms; r = 1, 310 x 301, lengths 400 and 361: 96 -> 8.9
// ms; wdtw r = 1, 500 x 403, length 256: 107 -> 9.0 ms.  Of the first, the
// sweep takes a third, the walk a fourth and the FP64 part two fifths (2100
// iterations for the 890 cells of a pair: lanes wait for the turn's longest
// word).

#include "guided.cuh"

#include <cfloat>
#include <cstdlib>

namespace wb {

namespace {

constexpr int kThreads = 128;
constexpr unsigned kCap = 1u << 30;  // saturated value, and out of band
constexpr int kFixOne = (1 << 29) - 1;  // 1.0 in fixed point

// Smallest and largest value of both series sets.  (The second is passed over
// only as the very same set: device arrays are used in place, so a set may
// start where the other does and hold more of it.)
__global__ void __launch_bounds__(256)
guided_range_kernel(const SeriesSet a, const SeriesSet b, GuidedPrep *prep) {
    double lo = WB_DBL_INF, hi = -WB_DBL_INF;
    for (int set = 0; set < 2; set++) {
        const SeriesSet &S = set ? b : a;
        if (set && b.base == a.base && b.stride == a.stride && b.len == a.len &&
            b.count == a.count)
            break;
        const int64_t total = S.count * (int64_t)S.len;
        for (int64_t t = (int64_t)blockIdx.x * 256 + threadIdx.x; t < total;
             t += (int64_t)gridDim.x * 256) {
            const int64_t s = t / S.len;
            double v = S.base[s * S.stride + (t - s * S.len)];
            if (isnan(v)) v = WB_DBL_INF;
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

// Float (value and rest) and 30-bit fixed-point copies of the centred, scaled
// series (one warp per series) with their extremes.  Row series start at element 3, which puts
// row 1 + S s on a 16-byte boundary.  Past a series' end the float copies cost
// +inf; the fixed-point ones hold 0 (cells there precede no cell of the
// pair).
__global__ void __launch_bounds__(256)
guided_convert_kernel(const SeriesSet rows, const SeriesSet cols, const GuidedSeries D,
                      const GuidedPrep *prep, const double *weights, int nw) {
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
        const int64_t at = s * (row ? D.xs : D.ys);
        float *dst = (row ? D.xf : D.yf) + at;
        int *dsq = row ? D.xq : D.yq;
        if (dsq) dsq += at;
        float *low = row ? D.xl : D.yl;
        if (low) low += at;
        double *as = row ? D.xd : D.yd;
        if (as) as += at;
        const int lead = row ? 3 : 0;
        const int total = (int)(row ? D.xs : D.ys);
        const float pad = row ? WB_FLT_INF : -WB_FLT_INF;
        float mx = 0.0f;
        int lo = kFixOne, hi = -kFixOne;
        for (int i = lane; i < total; i += 32) {
            const int e = i - lead;
            float v = pad, rest = 0.0f;
            int q = 0;
            double given = 0.0;
            if (e >= 0 && e < S.len) {
                given = src[e];
                const double c = (given - centre) * scale;
                v = (float)c;
                rest = (float)(c - (double)v);
                q = __double2int_rn(c * (double)kFixOne);
                mx = fmaxf(mx, fabsf(v));
                lo = imin(lo, q);
                hi = imax(hi, q);
            }
            dst[i] = v;
            if (dsq) dsq[i] = q;
            if (low) low[i] = rest;
            if (as) as[i] = given;
        }
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        lo = __reduce_min_sync(0xffffffffu, lo);
        hi = __reduce_max_sync(0xffffffffu, hi);
        if (lane == 0) (row ? D.xr : D.yr)[s] = GuidedRange{lo, hi, mx};
    }
    // weights by |i - j|, for i - j of either sign (a zero weight would turn an
    // infinite cost into NaN; 1e-38 is far below the bound's absolute term)
    if (D.wext)
        for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < D.wlen;
             i += (int64_t)gridDim.x * 256) {
            const int d = abs((int)i - D.woff);
            D.wext[i] = fmaxf((float)weights[d < nw ? d : nw - 1], FLT_MIN);
        }
}

// --------------------------------------------------------------------------

// ((a - b) + (al - bl))^2 of both halves
__device__ __forceinline__ void sqdiff2(uint64_t a, uint64_t al, uint64_t b, uint64_t bl,
                                        float &d0, float &d1) {
    asm("{\n\t.reg .b64 p, q;\n\tsub.rn.f32x2 p, %2, %4;\n\tsub.rn.f32x2 q, %3, %5;\n\t"
        "add.rn.f32x2 p, p, q;\n\tmul.rn.f32x2 p, p, p;\n\tmov.b64 {%0, %1}, p;\n\t}"
        : "=f"(d0), "=f"(d1)
        : "l"(a), "l"(al), "l"(b), "l"(bl));
}

// smallest predecessor (with the move's penalty) of a cell
template <int KIND>
__device__ __forceinline__ unsigned best_of(unsigned dg, unsigned up, unsigned lf, unsigned pen) {
    if constexpr (KIND == K_ADTW) return __viaddmin_u32(umin(up, lf), pen, dg);
    else return __vimin3_u32(dg, up, lf);
}

// best + cost in units, saturating, from a float square (the conversion
// saturates at 2^31 - 1)
template <int KIND>
__device__ __forceinline__ unsigned add_cost(float sq, float w, unsigned best) {
    if constexpr (KIND == K_WDTW) sq = __fmul_rn(sq, w);
    return __viaddmin_u32(best, (unsigned)__float2int_rn(sq), kCap);
}

// best + d^2 / 2^32 (rounded down), not saturating
__device__ __forceinline__ unsigned add_square(int d, unsigned best) {
    unsigned r;
    asm("mad.hi.s32 %0, %1, %1, %2;" : "=r"(r) : "r"(d), "r"(best));
    return r;
}

// A signed power of two as a left and a right shift (one of them 0), so that
// applying it takes two instructions and no choice.
struct Shift {
    int left, right;
    __device__ __forceinline__ int of(int x) const {
        return (int)((unsigned)x << left) >> right;
    }
};

// A pair's padded series and their scale: su for the float copies, a shift for
// the fixed-point ones.
struct PairData {
    const float *xf, *yf, *xl, *yl;
    const int *xq, *yq;
    float su;
    Shift shift;
    unsigned pen;
};

// The S rows of a strip or block from row i0: scaled float pairs with their
// low parts, or fixed point.
template <int S, bool FIX>
struct StripRows {
    uint64_t x2[S / 2], l2[S / 2];
    __device__ __forceinline__ void load(const PairData &D, int i0) {
        const float4 *x4 = reinterpret_cast<const float4 *>(D.xf + 3 + i0);
        const float4 *l4 = reinterpret_cast<const float4 *>(D.xl + 3 + i0);
#pragma unroll
        for (int k = 0; k < S / 4; k++) {
            const float4 t = x4[k], u = l4[k];
            x2[2 * k] = pack2(__fmul_rn(t.x, D.su), __fmul_rn(t.y, D.su));
            x2[2 * k + 1] = pack2(__fmul_rn(t.z, D.su), __fmul_rn(t.w, D.su));
            l2[2 * k] = pack2(__fmul_rn(u.x, D.su), __fmul_rn(u.y, D.su));
            l2[2 * k + 1] = pack2(__fmul_rn(u.z, D.su), __fmul_rn(u.w, D.su));
        }
    }
};
template <int S>
struct StripRows<S, true> {
    int x[S];
    __device__ __forceinline__ void load(const PairData &D, int i0) {
        const int4 *x4 = reinterpret_cast<const int4 *>(D.xq + 3 + i0);
#pragma unroll
        for (int k = 0; k < S / 4; k++) {
            const int4 t = x4[k];
            x[4 * k] = D.shift.of(t.x);
            x[4 * k + 1] = D.shift.of(t.y);
            x[4 * k + 2] = D.shift.of(t.z);
            x[4 * k + 3] = D.shift.of(t.w);
        }
    }
};

// Columns 4 g .. 4 g + 3, as loaded and scaled.
template <bool FIX>
struct Columns {
    uint4 v, l;
    __device__ __forceinline__ void load(const PairData &D, int g) {
        v = reinterpret_cast<const uint4 *>(FIX ? (const void *)D.yq : (const void *)D.yf)[g];
        if constexpr (!FIX) l = reinterpret_cast<const uint4 *>(D.yl)[g];
    }
    __device__ __forceinline__ unsigned one(const PairData &D, unsigned t) const {
        if constexpr (FIX) return (unsigned)D.shift.of((int)t);
        else return __float_as_uint(__fmul_rn(__uint_as_float(t), D.su));
    }
    __device__ __forceinline__ void scaled(const PairData &D, unsigned (&y)[4],
                                           unsigned (&yl)[4]) const {
        y[0] = one(D, v.x);
        y[1] = one(D, v.y);
        y[2] = one(D, v.z);
        y[3] = one(D, v.w);
        if constexpr (!FIX) {
            yl[0] = one(D, l.x);
            yl[1] = one(D, l.y);
            yl[2] = one(D, l.z);
            yl[3] = one(D, l.w);
        }
    }
};

// One column of a strip: Pin holds column c - 1, Pout receives column c;
// wq[S - 1 - k] is the weight of row k.  Fixed-point values saturate only at
// the end of a group of 4 columns: with squares of at most 2^28 (S = 8), or
// squares and penalties of at most 2^26, the S + 3 cells of a path through a
// group stay below 2^32.
template <int KIND, int S, bool FIX, bool MASK>
__device__ __forceinline__ void sweep_column(const unsigned (&Pin)[S], unsigned (&Pout)[S],
                                             unsigned bup, unsigned bdiag,
                                             const StripRows<S, FIX> &R, unsigned ybits,
                                             unsigned lbits, const float *wq, unsigned pen, unsigned M) {
    const float yf = __uint_as_float(ybits), lf = __uint_as_float(lbits);
    const uint64_t yy = FIX ? 0 : pack2(yf, yf), ll = FIX ? 0 : pack2(lf, lf);
#pragma unroll
    for (int k = 0; k < S; k += 2) {
        float sq[2];
        if constexpr (!FIX) sqdiff2(R.x2[k / 2], R.l2[k / 2], yy, ll, sq[0], sq[1]);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int i = k + h;
            const unsigned dg = i == 0 ? bdiag : Pin[i > 0 ? i - 1 : 0];
            const unsigned up = i == 0 ? bup : Pout[i > 0 ? i - 1 : 0];
            const unsigned best = best_of<KIND>(dg, up, Pin[i], pen);
            unsigned v;
            if constexpr (FIX) v = add_square(R.x[i] - (int)ybits, best);
            else v = add_cost<KIND>(sq[h], KIND == K_WDTW ? wq[S - 1 - i] : 1.0f, best);
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

// Step 1: the sweep; returns the value of cell (n-1, m-1) in units.  All lanes
// of a warp share the band.
template <int KIND, int S, bool FIX>
__device__ __forceinline__ unsigned guided_sweep(const GuidedArgs &A, const Band &B,
                                                 const PairData &D, int64_t gt) {
    constexpr int LG = S == 8 ? 1 : 2;  // groups of 4 columns per block, as a shift
    const int64_t nth = A.nth;
    const int G = A.groups, NB = A.blocks;
    const uint4 CAP4 = make_uint4(kCap, kCap, kCap, kCap);
    const unsigned pen = D.pen;
    unsigned result = kCap;
    // row 0: cumulative, without penalties, weight index j - 1
    {
        const float x0 = __fmul_rn(D.xf[3], D.su), x0l = __fmul_rn(D.xl[3], D.su);
        const int x0q = FIX ? D.shift.of(D.xq[3]) : 0;
        const int lim = imin(B.m, B.mx);
        unsigned acc = 0;
        for (int g = 0; g <= (lim - 1) >> 2; g++) {
            Columns<FIX> Y;
            Y.load(D, g);
            unsigned y[4], yl[4], v[4];
            Y.scaled(D, y, yl);
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int c = 4 * g + q;
                if constexpr (FIX) {
                    acc = umin(add_square(x0q - (int)y[q], acc), kCap);
                } else {
                    const float d = __fadd_rn(__fsub_rn(x0, __uint_as_float(y[q])),
                                              __fsub_rn(x0l, __uint_as_float(yl[q])));
                    const float w = KIND == K_WDTW ? A.wext[A.woff + imax(c - 1, 0)] : 1.0f;
                    acc = add_cost<KIND>(__fmul_rn(d, d), w, acc);
                }
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
        StripRows<S, FIX> R;
        R.load(D, i0);
        const uint4 *in = A.ckrow + ((int64_t)s * G - pg0) * nth + gt;
        uint4 *out = A.ckrow + ((int64_t)(s + 1) * G - g0) * nth + gt;
        uint4 *col = A.ckcol + ((int64_t)s * NB - (g0 >> LG)) * (S / 4) * nth + gt;
        auto up4 = [&](int g) { return g >= pg0 && g <= pg1 ? in[(int64_t)g * nth] : CAP4; };
        unsigned P[S], Q[S];
#pragma unroll
        for (int k = 0; k < S; k++) P[k] = kCap;
        unsigned bd = up4(g0 - 1).w;
        // the row above two groups ahead, the columns one
        uint4 nu = up4(g0), nnu = up4(g0 + 1);
        Columns<FIX> Y;
        Y.load(D, g0);
        for (int g = g0; g <= g1; g++) {
            const uint4 u = nu;
            unsigned y[4], yl[4];
            Y.scaled(D, y, yl);
            nu = nnu;
            nnu = up4(g + 2);
            if (g < g1) Y.load(D, g + 1);
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
                sweep_column<KIND, S, FIX, false>(P, Q, u.x, bd, R, y[0], yl[0], w, pen, 0u);
                o.x = Q[S - 1];
                sweep_column<KIND, S, FIX, false>(Q, P, u.y, u.x, R, y[1], yl[1], w + 1, pen, 0u);
                o.y = P[S - 1];
                sweep_column<KIND, S, FIX, false>(P, Q, u.z, u.y, R, y[2], yl[2], w + 2, pen, 0u);
                o.z = Q[S - 1];
                sweep_column<KIND, S, FIX, false>(Q, P, u.w, u.z, R, y[3], yl[3], w + 3, pen, 0u);
                o.w = P[S - 1];
            } else {
                const int e = 4 * g - i0 - B.lo;
                auto masked = [&](int q, const unsigned(&Pin)[S], unsigned(&Pout)[S],
                                  unsigned bup, unsigned bdg) {
                    const unsigned M = band_rows(e + q, B.width);
                    sweep_column<KIND, S, FIX, true>(Pin, Pout, bup, bdg, R, y[q], yl[q], w + q,
                                                     pen, M);
                    if (s == B.ns - 1 && 4 * g + q == B.m - 1) {
#pragma unroll
                        for (int k = 0; k < S; k++)
                            if (k < rows) result = Pout[k];
                    }
                };
                masked(0, P, Q, u.x, bd);
                o.x = Q[S - 1];
                masked(1, Q, P, u.y, u.x);
                o.y = P[S - 1];
                masked(2, P, Q, u.z, u.y);
                o.z = Q[S - 1];
                masked(3, Q, P, u.w, u.z);
                o.w = P[S - 1];
            }
            if constexpr (FIX) {
#pragma unroll
                for (int k = 0; k < S; k++) P[k] = umin(P[k], kCap);
                o = make_uint4(umin(o.x, kCap), umin(o.y, kCap), umin(o.z, kCap), P[S - 1]);
                result = umin(result, kCap);
            }
            bd = u.w;
            out[(int64_t)g * nth] = o;
            if (((g + 1) & ((1 << LG) - 1)) == 0) {
                uint4 *cd = col + (int64_t)(g >> LG) * (S / 4) * nth;
#pragma unroll
                for (int k = 0; k < S / 4; k++)
                    __stcs(cd + k * nth, make_uint4(P[4 * k], P[4 * k + 1], P[4 * k + 2],
                                                    P[4 * k + 3]));
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
template <int KIND, int S, bool FIX>
__device__ __forceinline__ void block_bits(const GuidedArgs &A, const Band &B, int s, int b,
                                           const PairData &D, int64_t gt, unsigned tol,
                                           unsigned (&xd)[S], unsigned (&xu)[S],
                                           unsigned (&xl)[S]) {
    constexpr int LG = S == 8 ? 1 : 2;
    const int64_t nth = A.nth;
    const int i0 = 1 + s * S, c0 = b * S;
    StripRows<S, FIX> R;
    R.load(D, i0);
    const unsigned pen = D.pen;
    unsigned P[S], Q[S], top[S], y[S], yl[S];
    float w[2 * S];
#pragma unroll
    for (int k = 0; k < S / 4; k++) {
        Columns<FIX> Y;
        Y.load(D, (c0 >> 2) + k);
        unsigned t[4], u[4];
        Y.scaled(D, t, u);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            y[4 * k + q] = t[q];
            if (!FIX) yl[4 * k + q] = u[q];
        }
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
        const float yf = __uint_as_float(y[q]), lf_ = FIX ? 0.0f : __uint_as_float(yl[q]);
        const uint64_t yy = FIX ? 0 : pack2(yf, yf), ll = FIX ? 0 : pack2(lf_, lf_);
        unsigned bd_ = 0, bu_ = 0, bl_ = 0;
#pragma unroll
        for (int k = 0; k < S; k += 2) {
            float sq[2];
            if constexpr (!FIX) sqdiff2(R.x2[k / 2], R.l2[k / 2], yy, ll, sq[0], sq[1]);
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int i = k + h, j = i > 0 ? i - 1 : 0;
                const unsigned dg = i == 0 ? (q == 0 ? bd : top[q > 0 ? q - 1 : 0]) : P[j];
                const unsigned up = i == 0 ? top[q] : Q[j];
                const unsigned lf = P[i];
                const unsigned best = best_of<KIND>(dg, up, lf, pen);
                // (saturated cells, those out of band among them, are never kept)
                const int t = (int)__viaddmin_u32(best, tol, kCap - 1u);
                const int tm = KIND == K_ADTW ? t - (int)pen : t;
                bd_ = push_sign(bd_, t - (int)dg);
                bu_ = push_sign(bu_, tm - (int)up);
                bl_ = push_sign(bl_, tm - (int)lf);
                unsigned v;
                if constexpr (FIX) v = umin(add_square(R.x[i] - (int)y[q], best), kCap);
                else v = add_cost<KIND>(sq[h], KIND == K_WDTW ? w[q - i + S - 1] : 1.0f, best);
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

// Steps 1 and 2 of the 32 pairs of a warp: the collected blocks go to the
// threads' lists (last block first); returns their number (-1: not collected)
// and in `row0` the last column collected of row 0.  e: the bound of an input
// difference's error in square roots of units.
template <int KIND, int S, bool FIX>
__device__ __forceinline__ int collect(const GuidedArgs &A, const Band &B, const PairData &D,
                                       float e, bool live, int64_t gt, int &row0) {
    constexpr int W64 = S * S / 64;  // mask words of a block
    constexpr unsigned SM = (1u << S) - 1u;
    const unsigned FULL = 0xffffffffu;
    const unsigned au = guided_sweep<KIND, S, FIX>(A, B, D, gt);

    // the bound (file header); sqrt(A_max) <= sqrt(A + K) (1 + 2^-22) + 2 e sqrt(K)
    const float K = (float)(B.n + B.m);
    const float ek = __fmul_ru(e, __fsqrt_ru(K));
    const float ra =
        __fmaf_ru(2.1f, ek, __fmul_ru(__fsqrt_ru(__fadd_ru((float)au, K)), 1.000001f));
    const float tolf = __fadd_ru(
        __fmaf_ru(KIND == K_ADTW ? 2.02f : 1.01f, K,
                  __fmul_ru(FIX ? (KIND == K_ADTW ? 4e-7f : 0.0f) : 1.2e-6f, __fmul_ru(ra, ra))),
        __fadd_ru(__fmul_ru(__fmul_ru(4.2f, ek), __fadd_ru(ra, ek)), 8.0f));
    live = live && au < kCap && tolf < 2.5e8f && __fadd_ru((float)au, tolf) < (float)kCap;
    const unsigned tol = live ? (unsigned)tolf : 0u;

    int s = B.ns - 1, b = (B.m - 1) / S;
    int slo = B.m - 1, shi = B.m - 1;  // seeds in the strip's bottom row
    int nlo = 0x7fffffff, nhi = -1;    // seeds of the strip above
    unsigned carry = 0;                // cells reached in the column left of the block
    int idx = live ? 0 : -1;
    while (__any_sync(FULL, live)) {
        if (live) {
            unsigned xd[S], xu[S], xl[S];
            block_bits<KIND, S, FIX>(A, B, s, b, D, gt, tol, xd, xu, xl);
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
            // (the last word first, like the blocks)
            uint4 *ent = A.list + (gt * A.list_cap + idx) * W64;
            const uint32_t pos = ((uint32_t)s << 16) | (uint32_t)b;
#pragma unroll
            for (int w = 0; w < W64; w++)
                ent[W64 - 1 - w] =
                    make_uint4(pos, (uint32_t)(mask[w] >> 32), (uint32_t)mask[w], 0u);
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
    row0 = shi;
    return idx;
}

// Step 3: the FP64 recurrence over the `count` collected blocks of each lane's
// pair (rows X, columns Y); the sum of cell (n-1, m-1), for lanes with
// count > 0.  The lanes go through their own blocks (mask words of 64 cells):
// a lane whose word is done takes the next one after the warp's turn of up to
// kCellsPerTurn cells, so the code that takes a word runs once per turn for
// the whole warp.  Longer turns idle more lanes, shorter ones take words more
// often: turns of 4, 6, 8 and 12 cells ran 1000 x 1000 pairs of length 512, r =
// 0.1 (other random walks), in 38.5, 38.2, 37.2 and 36.9 ms.
// Taking a word stages its rows, columns and the cells above it in shared
// memory (all loads in flight at once); a cell then waits for shared memory
// and the FP64 pipe only.  A lane's lists, bottom rows and series lie one after
// the other and are read 16 bytes at a time: with every value of a lane in a
// sector of its own (interleaved by thread) taking a word was 55 % of this
// step's time, now 37 %, and that call took 40.4 instead of 36.9 ms.  (An FP64 instruction takes 71 cycles of a warp and
// 21 of the SM whatever its active lanes, so what counts is the number of
// iterations: going through the strips in step, with the waits for the widest
// lane in each strip, measured 4.9 against 3.3 million cycles per 32 pairs of
// length 512.)
constexpr int kCellsPerTurn = 12;

template <int S>
struct Stage {
    static constexpr int C = 64 / S;  // columns of a mask word
    double value[S][kThreads];        // last value of every row
    double x[S][kThreads];
    double y[C][kThreads];
    double top[C + 1][kThreads];      // the row above, from the column left of the word
};

// Bits of a word's bottom row, column q in bit q.
template <int S>
__device__ __forceinline__ unsigned bottom_bits(uint64_t word) {
    constexpr int C = 64 / S;
    if constexpr (S == 8) {
        // bit 8 i to bit 56 + i: the products of distinct bits do not collide
        const uint64_t g = (word & 0x0101010101010101ull) * 0x0102040810204080ull;
        return __brev((unsigned)(g >> 56)) >> 24;
    }
    unsigned bits = 0;
#pragma unroll
    for (int q = 0; q < C; q++) bits |= (unsigned)((word >> (64 - S - q * S)) & 1u) << q;
    return bits;
}

// Whether the pairs to come go to the full recurrence at once: three quarters of
// `need` or more pairs were left or had a fourth of a wide band's blocks collected
// (values that tie everywhere).  `need` is half of the resident pairs, so that a few
// columns of such series among others decide nothing, and no job that the tail kernel
// takes.  dtw, length 512 (full recurrence / this): 1000 x 800 pairs, r = 0.1, spikes 237 /
// 230 ms (the second pass has its pairs dense), 0 / 1 values 237 / 183; r = 1, 500 x 400,
// spikes 319 / 328.
__device__ __forceinline__ bool ties_everywhere(const GuidedArgs &A) {
    const unsigned long long seen =
        *reinterpret_cast<const volatile unsigned long long *>(&A.prep->seen);
    const unsigned long long heavy =
        *reinterpret_cast<const volatile unsigned long long *>(&A.prep->heavy);
    return seen >= A.need && 4 * heavy >= 3 * seen;
}

// Whether the second pass comes anyway: pairs with more than a fourth of their blocks
// then go with it, also from under way (200 x 150 pairs of 256, r = 0.1, 0 / 1 values 4.3
// ms, without 4.8).
__device__ __forceinline__ bool second_pass_comes(const GuidedArgs &A) {
    return *reinterpret_cast<const volatile unsigned long long *>(&A.prep->heavy) >
           (unsigned long long)A.tail_cap;
}

// WATCH: a lane that is `large` ends without a value, count = -1, once
// second_pass_comes.  (Its own form: the test in the loop takes the others 0.7 % of the
// kernel's time.)
template <int KIND, int S, bool WATCH>
__device__ __forceinline__ double evaluate(const GuidedArgs &A, const double *__restrict__ X,
                                           const double *__restrict__ Y, int &count, int row0,
                                           int64_t gt, Stage<S> &St, bool large) {
    constexpr int W64 = S * S / 64;
    constexpr int C = 64 / S;
    constexpr unsigned SM = (1u << S) - 1u;
    constexpr unsigned TM = (1u << (C + 1)) - 1u;
    const double INF = WB_DBL_INF;
    const ElasticJob &J = A.J;
    const int tid = threadIdx.x;
    double *brow = A.brow + gt * 2 * A.brow_cols;  // [strip parity][column]: bottom rows
    const uint4 *list = A.list + gt * A.list_cap * W64;
    if (count > 0) {
        const double x0 = X[0];
        double acc = 0.0;
        for (int c = 0; c <= row0; c++) {
            const double v = x0 - __ldg(Y + c);
            double cst = v * v;
            if (KIND == K_WDTW) cst = cst * __ldg(J.weights + imax(c - 1, 0));
            acc = c == 0 ? cst : acc + cst;
            brow[c] = acc;
        }
    }
    // Of the strip above and of the current one: the words' columns, the first
    // word, and the collected cells of the bottom row (of 64 columns; the masks
    // are read again for wider strips).
    int pcol = 0, pend = 0, pfirst = 0;
    int ccol = 0, cend = 0, cfirst = 0;
    uint64_t pbits = 0, cbits = 0;
    int cur = -1, i0 = 0, cw = 0;
    double *below = brow;
    uint64_t M = 0, LM = 0, todo = 0;
    unsigned tops = 0;  // bit q: cell (i0 - 1, cw - 1 + q) is collected
    double last = 0.0, last_old = 0.0;
    int left = imax(count, 0) * W64;  // mask words to go
    // the next word, loaded while the current one is worked on
    uint4 next = left > 0 ? list[left - 1] : make_uint4(0u, 0u, 0u, 0u);
    while (__any_sync(0xffffffffu, todo != 0 || left > 0)) {
        if (todo == 0 && left > 0) {
            left--;
            if (WATCH && large && (left & 15) == 15 && second_pass_comes(A)) {
                left = 0;
                count = -1;
                continue;
            }
            const uint4 E = next;
            if (left > 0) next = list[left - 1];
            const int w = W64 - 1 - left % W64;
            const int bs = (int)(E.x >> 16), bb = (int)(E.x & 0xffffu);
            unsigned lm = (unsigned)(M & SM);  // collected rows of the column to the left
            M = ((uint64_t)E.y << 32) | E.z;
            cw = bb * S + w * C;
#pragma unroll
            for (int q = 0; q < C; q += 2) {
                const double2 v = __ldg(reinterpret_cast<const double2 *>(Y + cw + q));
                St.y[q][tid] = v.x;
                St.y[q + 1][tid] = v.y;
            }
            if (bs != cur) {
                pcol = ccol;
                pend = cend;
                pfirst = cfirst;
                pbits = cbits;
                ccol = cw;
                cfirst = left;
                cbits = 0;
                lm = 0;
                i0 = 1 + bs * S;
                below = brow + ((bs + 1) & 1) * A.brow_cols;
#pragma unroll
                for (int k = 0; k < S; k += 2) {
                    const double2 v = __ldg(reinterpret_cast<const double2 *>(X + i0 + k));
                    St.x[k][tid] = v.x;
                    St.x[k + 1][tid] = v.y;
                }
            }
            cend = cw + C;
            if (cw - ccol < 64) cbits |= (uint64_t)bottom_bits<S>(M) << (cw - ccol);
            LM = (M >> S) | ((uint64_t)lm << (64 - S));
            todo = M;
            // the cells above the word: row 0, or the bottom row of the strip
            // above
            if (bs == 0) {
                const int cells = row0 - cw + 2;
                tops = cells <= 0 ? 0u : cells > C ? TM : (1u << cells) - 1u;
                if (cw == 0) tops &= ~1u;
            } else if (pend - pcol <= 64) {
                const int sh = cw - 1 - pcol;
                tops = sh >= 64 || sh < -C ? 0u
                                           : (unsigned)(sh >= 0 ? pbits >> sh : pbits << -sh) & TM;
            } else {
                tops = 0;
#pragma unroll
                for (int o = 0; o < 2; o++) {  // the word's columns, those to the left
                    const int col = cw - o * C;
                    if (col < pcol || col >= pend) continue;
                    const uint4 v = list[pfirst - (col - pcol) / C];
                    const unsigned bits = bottom_bits<S>(((uint64_t)v.y << 32) | v.z);
                    tops |= o == 0 ? bits << 1 : bits >> (C - 1);
                }
            }
            const double *above = brow + (bs & 1) * A.brow_cols + cw;
            if (tops > 1u) {
#pragma unroll
                for (int q = 0; q < C; q += 2) {
                    const double2 v = *reinterpret_cast<const double2 *>(above + q);
                    St.top[q + 1][tid] = v.x;
                    St.top[q + 2][tid] = v.y;
                }
            }
            if (tops & 1u) St.top[0][tid] = above[-1];
            cur = bs;
        }
#pragma unroll 1
        for (int turn = 0; turn < kCellsPerTurn; turn++) {
            if (todo == 0) break;
            const int p = __clzll((long long)todo);
            const uint64_t bit = 0x8000000000000000ULL >> p;
            todo ^= bit;
            const int k = p & (S - 1), q = p / S;
            const double d = St.x[k][tid] - St.y[q][tid];
            double cst = d * d;
            if (KIND == K_WDTW) cst = cst * __ldg(J.weights + abs(i0 + k - cw - q));
            const double old = St.value[k][tid];
            const double lf = (LM & bit) ? old : INF;
            // above: the cell before in this column, or the row above the block
            const bool hu = k > 0 ? (M & (bit << 1)) != 0 : (tops >> (q + 1)) & 1u;
            const bool hd = k > 0 ? (LM & (bit << 1)) != 0 : (tops >> q) & 1u;
            const double tu = k > 0 ? last : St.top[q + 1][tid];
            const double td = k > 0 ? (hu ? last_old : St.value[k - 1][tid]) : St.top[q][tid];
            double mv = nn_min(hu ? tu : INF, lf);
            if (KIND == K_ADTW) mv = mv + J.p;
            const double nv = nn_min(mv, hd ? td : INF) + cst;
            St.value[k][tid] = nv;
            last = nv;
            last_old = old;
            if (k == S - 1) below[cw + q] = nv;
        }
    }
    return last;
}

template <int KIND, int S>
__global__ void __launch_bounds__(kThreads, S == 8 ? 4 : 3)
guided_pairs_kernel(const GuidedArgs A) {
    __shared__ Stage<S> stage;
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int64_t gt = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    const ElasticJob &J = A.J;
    const Band B(J, S);
    double centre = 0.0, scale = 1.0;
    const bool finite = centre_scale(A.prep, centre, scale);
    const float penf = KIND == K_ADTW ? __double2float_ru(J.p * scale * scale) : 0.0f;
    const int64_t chunks = (J.rows.count + 31) >> 5;
    const bool listed = A.items != nullptr || A.n_all > 0;
    const int64_t nlist = A.items ? (int64_t)*A.n_items : A.n_all;
    const int64_t ntiles = listed ? (nlist + 31) >> 5
                                  : (J.mode == PM_PAIRED ? chunks : chunks * J.cols.count);
    const float K = (float)(B.n + B.m);

    for (;;) {
        unsigned long long t64 = 0;
        bool give_up = false;
        if (lane == 0) {
            t64 = atomicAdd(&A.prep->queue, 1ull);
            give_up = ties_everywhere(A);
        }
        const int64_t t = (int64_t)__shfl_sync(FULL, t64, 0);
        if (t >= ntiles) break;
        int64_t cs = t / chunks;
        int64_t rs = (t - cs * chunks) * 32 + lane;
        if (J.mode == PM_PAIRED) {
            rs = t * 32 + lane;
            cs = rs;
        }
        bool active = rs < J.rows.count && !(J.mode == PM_UPPER && rs >= cs);
        if (listed) {
            const int64_t at = t * 32 + lane;
            active = at < nlist;
            const int64_t p = active ? (A.items ? (int64_t)A.items[at] : at) : 0;
            cs = A.col0 + p / J.rows.count;
            rs = p % J.rows.count;
        }
        if (!__any_sync(FULL, active)) continue;
        auto store = [&](double res) {
            if (J.mode == PM_PAIRED) {
                J.out[rs] = res;
            } else {
                J.out[rs * J.out_ld + cs] = res;
                if (J.mode == PM_UPPER) J.out[cs * J.out_ld + rs] = res;
            }
        };
        // the tile's pairs `who` to the second pass
        auto leave = [&](bool who) {
            const unsigned mask = __ballot_sync(FULL, who);
            if (mask == 0) return;
            unsigned long long at = 0;
            if (lane == 0) at = atomicAdd(&A.prep->pending, (unsigned long long)__popc(mask));
            at = __shfl_sync(FULL, at, 0) + __popc(mask & ((1u << lane) - 1u));
            if (!who) return;
            store(__longlong_as_double(kGuidedPending));
            if ((int64_t)at < A.left_cap)
                A.left[at] = J.mode == PM_PAIRED ? rs : rs + J.rows.count * cs;
        };
        if (__any_sync(FULL, give_up)) {
            leave(active);
            if (lane == 0) {
                atomicAdd(&A.prep->heavy, 32ull);
                atomicAdd(&A.prep->seen, 32ull);
            }
            continue;
        }
        if (!active && !listed) {  // sweeps along on a valid pair
            rs = J.rows.count - 1;
            cs = J.mode == PM_PAIRED ? rs : cs;
        }
        PairData D;
        D.xf = A.xf + rs * A.xs;
        D.yf = A.yf + cs * A.ys;
        D.xl = A.xl + rs * A.xs;
        D.yl = A.yl + cs * A.ys;
        D.xq = A.xq + rs * A.xs;
        D.yq = A.yq + cs * A.ys;
        const GuidedRange rx = A.xr[rs], ry = A.yr[cs];
        // upper bound of the sum (of the FP64 inputs too)
        float e = __fmaf_ru(6.0e-8f, __fadd_ru(rx.mag, ry.mag), 1e-37f);
        float ub = __fsqrt_ru(straight_path<KIND>(A, B, D.xf, D.yf, penf));
        ub = __fmaf_ru(e, __fsqrt_ru(K), ub);
        // (from 2^-97 on units are at most 2^124, so that a penalty of 0 stays 0)
        ub = fmaxf(__fmul_ru(ub, ub), 0x1p-97f);
        const bool live = active && finite && ub < 1e30f;
        const int lub = ilogbf(ub);
        // Fixed point: units of d^2 2^(26 + 2k) (d the scaled difference), the
        // shift k as large as the pair's largest difference (see sweep_column)
        // and the upper bound allow; where that
        // leaves too few units for the sums' K roundings (differences far
        // larger than the distance), the warp sweeps with float costs.
        bool fix = false;
        int shift = 0;
        float units = 0.0f;
        if constexpr (KIND != K_WDTW) {
            const int dmax = imax(imax(rx.hi - ry.lo, ry.hi - rx.lo), 1);
            const int bits = S == 8 && KIND == K_DTW ? 30 : 29;
            shift = imax(imin(bits - (32 - __clz(dmax)), (2 - lub) >> 1), -24);
            units = live ? scalbnf(1.0f, 26 + 2 * shift) : 0.0f;
            fix = __all_sync(FULL, !live || (ub * units >= 16384.0f * K &&
                                             penf * units <= 67108864.0f));
        }
        D.shift = Shift{imax(shift, 0), imax(-shift, 0)};
        const int half = live ? (28 - lub) >> 1 : 0;
        D.su = scalbnf(1.0f, half);
        if (fix) e = __fadd_ru(scalbnf(1.0f, shift), shift < 0 ? 2.0f : 0.0f) / 65536.0f;
        // (float differences with their low parts: relative errors apart,
        // which the bound counts, they are off by 2^-47 of the values)
        else e = __fmul_ru(__fmul_ru(e, 1.3e-7f), D.su);
        if (!fix) units = __fmul_rn(D.su, D.su);
        D.pen = KIND == K_ADTW
                    ? (unsigned)__float2int_rn(fminf(__fmul_rn(penf, units), (float)kCap))
                    : 0u;
        int row0 = -1, count;
        if (KIND != K_WDTW && fix) count = collect<KIND, S, KIND != K_WDTW>(A, B, D, e, live, gt, row0);
        else count = collect<KIND, S, false>(A, B, D, e, live, gt, row0);

        const bool large = 4 * count > B.ns * A.blocks;
        const unsigned heavy =
            __ballot_sync(FULL, active && (count <= 0 || (A.blocks >= 12 && large)));
        const int pairs = __popc(__ballot_sync(FULL, active));
        if (lane == 0) {
            if (heavy) atomicAdd(&A.prep->heavy, (unsigned long long)__popc(heavy));
            atomicAdd(&A.prep->seen, (unsigned long long)pairs);
        }

        double value = 0.0;
        if (large && second_pass_comes(A)) count = -1;
        const double *X = A.xd + rs * A.xs + 3, *Y = A.yd + cs * A.ys;
        if (__any_sync(FULL, large && count > 0))
            value = evaluate<KIND, S, true>(A, X, Y, count, row0, gt, stage, large);
        else if (__any_sync(FULL, count > 0))
            value = evaluate<KIND, S, false>(A, X, Y, count, row0, gt, stage, false);
        if (active && count > 0) store(sqrt(value));
        leave(active && count <= 0);
    }
}

// --------------------------------------------------------------------------
// Few pairs left over: the full recurrence of a pair on the 32 lanes of a warp,
// lane l on strips l, l + 32, .. of 8 rows, one column per step and one behind lane
// l - 1, whose bottom cell it takes by shuffle (lane 0: from a row in memory that
// lane 31 wrote); the cells' operations are the strip kernel's.  One thread per
// pair, as the second pass has them, takes 330 cycles for every cell: a single
// pair of 400 x 361, r = 1, kept the call waiting for 13 ms, here 1.
constexpr int kTailRows = 8;

template <int KIND>
__global__ void __launch_bounds__(kThreads) guided_tail_kernel(const GuidedArgs A) {
    constexpr int S = kTailRows, G = 32;
    const unsigned FULL = 0xffffffffu;
    const ElasticJob &J = A.J;
    const unsigned long long left = A.prep->pending;
    if (left == 0 || left > (unsigned long long)A.tail_cap) return;
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * kThreads + threadIdx.x) >> 5;
    const int64_t warps = ((int64_t)gridDim.x * kThreads) >> 5;
    double *row = A.brow + warp * A.brow_cols;
    const Band B(J, S);
    const int n = B.n, m = B.m, lim = imin(m, B.mx);
    const double INF = WB_DBL_INF;
    const int strips = B.ns;
    // steps from a round to the next: every lane is done with its strip and its
    // row is written a step before lane 0 reads it
    const int delta = imax(G + 2, imin(m, S + B.mx + B.mn + B.r - 2 - G * S));
    const int steps = (strips - 1) / G * delta + ((strips - 1) & (G - 1)) + m;
    for (int64_t q = warp; q < (int64_t)left; q += warps) {
        int64_t r1 = (int64_t)A.left[q], c1 = r1;
        if (J.mode != PM_PAIRED) {
            c1 = r1 / J.rows.count;
            r1 -= c1 * J.rows.count;
        }
        const double *X = J.rows.base + r1 * J.rows.stride;
        const double *Y = J.cols.base + c1 * J.cols.stride;
        double P[S], x[S], result = 0.0, acc = 0.0, bot = INF, bdiag = INF, before = INF;
#pragma unroll
        for (int k = 0; k < S; k++) P[k] = INF, x[k] = 0.0;
        const double x0 = X[0];
        int s = lane, c = -lane;
        for (int t = 0; t < steps; t++) {
            const double above = __shfl_up_sync(FULL, bot, 1);
            const bool any = s < strips;
            const int i0 = 1 + s * S;
            const int first = any ? B.cs(s, S) : m, end = any ? B.ce(s, S) : m;
            const int pfirst = any ? B.cs(s - 1, S) : 0, pend = any ? B.ce(s - 1, S) : 0;
            double up = above;
            if (lane == 0 && any) {
                up = INF;
                if (s > 0) {
                    if (c >= pfirst && c < pend) up = row[c];
                } else if (c < lim) {
                    const double v = x0 - __ldg(Y + c);
                    double cst = v * v;
                    if (KIND == K_WDTW) cst = cst * __ldg(J.weights + imax(c - 1, 0));
                    acc = c == 0 ? cst : acc + cst;
                    up = acc;
                }
            }
            const double raw = up;
            if (any && c >= first) {
                if (c == first) {
                    bdiag = INF;
                    if (c > pfirst && c <= pend) {
                        bdiag = before;
                        if (lane == 0 && s > 0) bdiag = row[c - 1];
                    }
#pragma unroll
                    for (int k = 0; k < S; k++) {
                        P[k] = INF;
                        x[k] = X[imin(i0 + k, n - 1)];
                    }
                }
                if (c >= pend) up = INF;
                const double y = __ldg(Y + c), above_cell = up;
                double dg = bdiag;
#pragma unroll
                for (int k = 0; k < S; k++) {
                    const int d = c - (i0 + k);
                    const double lf = P[k], v = x[k] - y;
                    double cst = v * v;
                    if (KIND == K_WDTW)
                        cst = cst * __ldg(J.weights + abs(c - imin(i0 + k, n - 1)));
                    double mv = nn_min(up, lf);
                    if (KIND == K_ADTW) mv = mv + J.p;
                    double nv = nn_min(mv, dg) + cst;
                    if (d < B.lo || d > B.mx - 1) nv = INF;
                    dg = lf;
                    up = nv;
                    P[k] = nv;
                }
                bot = P[S - 1];
                bdiag = above_cell;
                if (lane == G - 1 && s + 1 < strips) row[c] = bot;
                if (s == strips - 1 && c == m - 1) {
#pragma unroll
                    for (int k = 0; k < S; k++)
                        if (i0 + k < n) result = P[k];
                }
            }
            before = raw;
            c++;
            if (any && c >= end) {
                s += G;
                c -= delta;
            }
            __syncwarp();
        }
        const double v = sqrt(__shfl_sync(FULL, result, (strips - 1) & (G - 1)));
        if (lane == 0) {
            if (J.mode == PM_PAIRED) {
                J.out[r1] = v;
            } else {
                J.out[r1 * J.out_ld + c1] = v;
                if (J.mode == PM_UPPER) J.out[c1 * J.out_ld + r1] = v;
            }
        }
        __syncwarp();
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
    int64_t left_cap = 0;     // entries of the list of pairs left
    int64_t tail_cap = 0;     // most pairs left that guided_tail_kernel takes
    size_t shared_bytes = 0;  // copies of the series, their extremes, weights, prep
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

// Budget of the kept rows and columns of all resident pairs, for blocks of 8
// cells and of 16.  Where 8 cells need more, their rows and columns bound the
// kernel by DRAM writes (310 x 301 pairs of 400 x 361, r = 1: 2.2 ms more with 12 GB
// than the 8.1 to 9.3 of blocks of 16); blocks of 16 are worth every resident warp (600 x 500
// pairs of 900, r = 0.2, 14 GB: 84 -> 71 ms against the 62 % that 8 GB hold).
constexpr size_t kGuidedBudget8 = (size_t)8 << 30;
constexpr size_t kGuidedBudget16 = (size_t)16 << 30;

// Pairs left that guided_tail_kernel takes: as long as its FP64 instructions (24 a
// step, 21 cycles of an SM each) take no longer than a thread of the second pass
// takes for its pair (330 cycles a cell), halved.  2200 of 256 x 256, r = 0.1.
int64_t tail_pairs(int n, int m, int r) {
    const int64_t width = imin(m, imax(0, m - n) + imax(0, n - m) + 2 * r - 1);
    const int64_t strips = (n - 1 + kTailRows - 1) / kTailRows;
    const int64_t delta = imax(34, imin(m, (int)width + r));
    const int64_t steps = (strips - 1) / 32 * delta + 31 + m;
    return std::max<int64_t>(256, device_info().sm_count * n * width / 3 / steps);
}

// More pairs left than this are found by their outputs, tile by tile.
constexpr int64_t kLeftCap = (int64_t)1 << 25;

// max_pairs > 0: for lists of at most so many pairs
Plan plan_guided(const ElasticJob &J, size_t avail, int64_t max_pairs = 0) {
    Plan p;
    const int n = J.rows.len, m = J.cols.len, r = J.band;
    if (J.kind != K_DTW && J.kind != K_WDTW && J.kind != K_ADTW) return p;
    if ((J.key && max_pairs == 0) || J.all_zero || J.pending) return p;
    if (J.mode == PM_UPPER && J.rows.count < 2) return p;  // no pairs
    const char *e = getenv("WB_GPU_ELASTIC");
    if (e && (strcmp(e, "ring") == 0 || strcmp(e, "strip") == 0)) return p;
    const int mx = imax(0, m - n) + r, mn = imax(0, n - m);
    const int width = mx + mn + r - 1;
    if (imin(n, m) < 24 || imin(width, m) < 12) return p;
    if ((int64_t)n + m > 1 << 15) return p;  // positions are 16 bits
    const DeviceInfo &dev = device_info();
    int64_t work = (J.mode == PM_PAIRED ? (J.rows.count + 31) / 32
                                        : (J.rows.count + 31) / 32 * J.cols.count) * 32;
    if (max_pairs > 0) work = std::min(work, max_pairs);
    p.tail_cap = std::min(work, tail_pairs(n, m, r));
    // (a list's second pass finds its pairs by their outputs)
    p.left_cap = max_pairs > 0 ? p.tail_cap : std::min<int64_t>(work, kLeftCap);
    // wdtw between very unequal lengths: the path ends on a diagonal whose weight
    // is up to 10^10 times that of the main one, near which cells cost less than
    // the 32-bit resolution and are all collected.  With two warps per SM their
    // FP64 latency decides: 60 x 50 pairs of 60 and 900 take 19.7 ms, the full
    // recurrence 10.0 (200 and 300: 2.8 and 9.5; 231 x 34 of 527 and 375: 13.9
    // and 15.5; with four times the pairs 16.3 and 26.6).
    if (J.kind == K_WDTW && imax(n, m) >= 640 && 2 * std::abs(n - m) >= imax(n, m) &&
        work <= 64 * dev.sm_count)
        return p;
    const int64_t want = (work + kThreads - 1) / kThreads;
    for (int S = 8; S <= 16; S += 8) {
        const int ns = (n - 1 + S - 1) / S;
        p.S = S;
        p.groups = (imin(m, width + S - 1) + 3) / 4 + 1;
        p.blocks = p.groups / (S / 4) + 2;
        // a wide band's pairs with more of its blocks are faster in guided_tail_kernel or
        // the second pass; 600 x 500 pairs of 900, r = 0.2: 58 to 61 ms, with half of
        // them 64 to 102, waiting for one pair (narrow bands: 200 x 150 pairs of 256, r =
        // 0.1, noise 1.6 ms with half, 1.9 with a fourth)
        p.list_cap = imax((n + m) / S + 8, ns * p.blocks / (p.blocks < 12 ? 2 : 4));
        p.brow_cols = (int)round_up(m, S);
        p.xs = round_up(3 + 1 + (int64_t)ns * S, 4);
        p.ys = round_up(m, 16);
        p.woff = (int)round_up(n + 2 * S, 4);
        p.wlen = J.kind == K_WDTW ? (int)round_up(p.woff + m + 2 * S, 4) : 0;
        p.thread_bytes = (size_t)(ns + 1) * p.groups * 16 + (size_t)ns * p.blocks * S * 4 +
                         (size_t)p.list_cap * (S * S / 64) * 16 + (size_t)2 * p.brow_cols * 8;
        p.shared_bytes = 3 * align256(J.rows.count * p.xs * 4) +
                         3 * align256(J.cols.count * p.ys * 4) +
                         align256(J.rows.count * p.xs * 8) + align256(J.cols.count * p.ys * 8) +
                         align256(J.rows.count * sizeof(GuidedRange)) +
                         align256(J.cols.count * sizeof(GuidedRange)) +
                         align256((size_t)imax(p.wlen, 1) * 4) + align256(sizeof(GuidedPrep)) +
                         align256((size_t)p.left_cap * 8) + 4 * 256;
        int nb;
        switch (J.kind) {
            case K_DTW: nb = blocks_per_sm<K_DTW>(S); break;
            case K_WDTW: nb = blocks_per_sm<K_WDTW>(S); break;
            default: nb = blocks_per_sm<K_ADTW>(S); break;
        }
        const int64_t full = std::min<int64_t>(want, (int64_t)imax(nb, 1) * dev.sm_count);
        const size_t room = std::min(S == 8 ? kGuidedBudget8 : kGuidedBudget16,
                                     avail > p.shared_bytes ? avail - p.shared_bytes : 0);
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
int run_kernel(const GuidedContext &C, cudaStream_t s) {
    if (C.S == 8) guided_pairs_kernel<KIND, 8><<<C.grid, kThreads, 0, s>>>(C.args);
    else guided_pairs_kernel<KIND, 16><<<C.grid, kThreads, 0, s>>>(C.args);
    WB_LAUNCH_CHECK("guided_pairs_kernel");
    return WB_OK;
}

int run_tail(const GuidedContext &C, cudaStream_t s) {
    // a warp per pair: at most half the rows of `brow`
    const int grid = (int)std::min<int64_t>(
        {(C.args.tail_cap + 3) / 4, C.args.nth / 4, (int64_t)16 * device_info().sm_count});
    switch (C.args.J.kind) {
        case K_DTW: guided_tail_kernel<K_DTW><<<grid, kThreads, 0, s>>>(C.args); break;
        case K_WDTW: guided_tail_kernel<K_WDTW><<<grid, kThreads, 0, s>>>(C.args); break;
        default: guided_tail_kernel<K_ADTW><<<grid, kThreads, 0, s>>>(C.args); break;
    }
    WB_LAUNCH_CHECK("guided_tail_kernel");
    return WB_OK;
}

}  // namespace

static size_t plan_bytes(const Plan &p) {
    return p.use ? p.shared_bytes + 2 * 4096 + p.thread_bytes * (size_t)p.grid * kThreads : 0;
}

size_t guided_workspace_bytes(const ElasticJob &J) {
    if (bit_edit_supported(J)) return bit_edit_bytes(J);
    if (wave_supported(J)) {
        const size_t own = wave_bytes(J), other = elastic_workspace_bytes(J);
        return own > other ? own - other : 0;
    }
    return plan_bytes(plan_guided(J, SIZE_MAX));
}

size_t guided_list_bytes(const ElasticJob &J, int64_t max_pairs) {
    return plan_bytes(plan_guided(J, SIZE_MAX, max_pairs));
}

int guided_series(const ElasticJob &J, const GuidedSeries &S, GuidedPrep *prep, cudaStream_t s) {
    // lo = a very large code, hi = a very small one
    WB_CUDA(cudaMemsetAsync(&prep->lo, 0x7f, sizeof(prep->lo), s));
    WB_CUDA(cudaMemsetAsync(&prep->hi, 0x80, sizeof(prep->hi), s));
    const int64_t cap = (int64_t)device_info().sm_count * 4;
    const int64_t values = J.rows.count * J.rows.len + J.cols.count * J.cols.len;
    guided_range_kernel<<<(int)std::min(cap, (values + 1023) / 1024), 256, 0, s>>>(
        J.rows, J.cols, prep);
    WB_LAUNCH_CHECK("guided_range_kernel");
    const int64_t series = J.rows.count + J.cols.count;
    guided_convert_kernel<<<(int)std::min(cap, (series + 7) / 8), 256, 0, s>>>(
        J.rows, J.cols, S, prep, J.weights, S.wext ? imax(J.rows.len, J.cols.len) : 0);
    WB_LAUNCH_CHECK("guided_convert_kernel");
    return WB_OK;
}

int guided_prepare(const ElasticJob &J, Workspace &ws, size_t leave, int64_t max_pairs,
                   GuidedContext &C) {
    leave += 4096;  // and the alignment of the pieces
    const size_t avail = ws.remaining();
    const Plan p = plan_guided(J, avail > leave ? avail - leave : 0, max_pairs);
    C.args.prep = nullptr;
    if (!p.use) return WB_OK;
    cudaStream_t s = ws.stream();
    const int ns = (J.rows.len - 1 + p.S - 1) / p.S;
    const int64_t nth = (int64_t)p.grid * kThreads;
    C.S = p.S;
    C.grid = p.grid;
    GuidedArgs &A = C.args;
    A.J = J;
    A.nth = nth;
    A.need = (unsigned)std::max<int64_t>(p.tail_cap, nth / 2);
    A.tail_cap = p.tail_cap;
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
    WB_TAKE(xl, float, ws, J.rows.count * p.xs);
    WB_TAKE(yl, float, ws, J.cols.count * p.ys);
    WB_TAKE(xq, int, ws, J.rows.count * p.xs);
    WB_TAKE(yq, int, ws, J.cols.count * p.ys);
    WB_TAKE(xd, double, ws, J.rows.count * p.xs);
    WB_TAKE(yd, double, ws, J.cols.count * p.ys);
    WB_TAKE(xr, GuidedRange, ws, J.rows.count);
    WB_TAKE(yr, GuidedRange, ws, J.cols.count);
    WB_TAKE(wext, float, ws, imax(p.wlen, 1));
    WB_TAKE(ckrow, uint4, ws, (size_t)(ns + 1) * p.groups * nth);
    WB_TAKE(ckcol, uint4, ws, (size_t)ns * p.blocks * (p.S / 4) * nth);
    WB_TAKE(list, uint4, ws, (size_t)p.list_cap * (p.S * p.S / 64) * nth);
    WB_TAKE(brow, double, ws, (size_t)2 * p.brow_cols * nth);
    if (p.left_cap > 0) {
        WB_TAKE(left, unsigned long long, ws, (size_t)p.left_cap);
        A.left = left;
        A.left_cap = p.left_cap;
    }
    A.prep = prep;
    A.xf = xf;
    A.yf = yf;
    A.xl = xl;
    A.yl = yl;
    A.xq = xq;
    A.yq = yq;
    A.xd = xd;
    A.yd = yd;
    A.xr = xr;
    A.yr = yr;
    A.wext = wext;
    A.ckrow = ckrow;
    A.ckcol = ckcol;
    A.list = list;
    A.brow = brow;
    GuidedSeries S;
    S.xf = xf;
    S.yf = yf;
    S.xl = xl;
    S.yl = yl;
    S.xq = xq;
    S.yq = yq;
    S.xd = xd;
    S.yd = yd;
    S.xs = p.xs;
    S.ys = p.ys;
    S.xr = xr;
    S.yr = yr;
    if (p.wlen) {
        S.wext = wext;
        S.woff = p.woff;
        S.wlen = p.wlen;
    }
    WB_TRY(guided_series(J, S, prep, s));
    return WB_OK;
}

int guided_run(const GuidedContext &C, cudaStream_t s) {
    GuidedPrep *prep = C.args.prep;
    WB_CUDA(cudaMemsetAsync(&prep->queue, 0, 4 * sizeof(unsigned long long), s));
    switch (C.args.J.kind) {
        case K_DTW: WB_TRY(run_kernel<K_DTW>(C, s)); break;
        case K_WDTW: WB_TRY(run_kernel<K_WDTW>(C, s)); break;
        default: WB_TRY(run_kernel<K_ADTW>(C, s));
    }
    return run_tail(C, s);
}

int launch_guided(ElasticJob &J, Workspace &ws, size_t leave) {
    GuidedContext C;
    WB_TRY(guided_prepare(J, ws, leave, 0, C));
    if (!C.args.prep) return WB_OK;
    timer_begin("guided_pairs_kernel", ws.stream());
    WB_TRY(guided_run(C, ws.stream()));
    timer_end(ws.stream());
    J.pending = &C.args.prep->pending;
    J.left = C.args.left;
    J.left_cap = C.args.left_cap;
    J.tail_cap = C.args.tail_cap;
    return WB_OK;
}

}  // namespace wb
