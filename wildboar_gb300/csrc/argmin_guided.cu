// argmin_guided.cu -- argmin_distance of the dtw family (dtw, wdtw, ddtw,
// wddtw, adtw with a penalty >= 0) with float32 bounds in front of the guided
// FP64 evaluation (guided.cu).
//
// The reference walks a query's candidates in order and keeps a k-max-heap;
// candidate j changes it only if its distance is below the heap's k-th
// distance at that point (Heap.push replaces the root only by a smaller
// value).  For these metrics early abandoning never decides that: the abandon
// key (the largest row minimum) is at most the final sum v, since costs and
// penalties are not negative and rounding is monotone, and key > fl(D D)
// implies v > fl(D D), hence sqrt(v) >= D: the candidate would not have been
// pushed either.  The k-th distance only decreases, so a candidate of a chunk
// whose distance exceeds the k-th distance D after the chunks before it can
// be dropped; its place is filled with +inf.
//
// Candidates go in chunks that grow by kGrowth.  In each chunk
//   1. lb_filter_kernel drops pairs by LB_Keogh in float32 (the query's
//      values against the candidate's envelope over the band; one thread per
//      query and kLbCols candidates, query values coalesced, envelopes
//      broadcast);
//   2. sweep_filter_kernel runs the band recurrence in float32 over the pairs
//      left and drops them at the first strip of rows whose bottom row lies
//      above the bound;
//   3. the guided evaluation gives the exact distance of the rest;
//   4. the heap replay advances over the chunk (argmin.cu).
// Both filters compare float sums with the bound
//   (sqrt(D^2) + e sqrt(K))^2 (1 + g),
// K = n + m, e = 2^-24 (max|x| + max|y|) the rounding of the inputs, g the
// roundings of at most 2 K + 16 operations, all rounded up: a pair dropped has
// an FP64 distance above D.  Fast paths never accept, they only drop.
//
// Measured on one GB300, 500 queries x 2000 random walks of length 512,
// r = 0.1, k = 5: 162 ms (FP64 in early-abandoned chunks) -> 10.5 ms, of which
// the three guided evaluations take 6, the float sweeps 1.5 and LB_Keogh 0.3 ms.

#include "guided.cuh"

#include <cfloat>
#include <cstdlib>

#include "argmin.cuh"

namespace wb {

namespace {

constexpr int kLbCols = 4;      // candidates per thread of the first filter
constexpr int kLbMaxLen = 4096; // envelopes are built in shared memory

// Envelope of every column series over the columns in band of each row:
// env[j][i] = (min, max) of y_j over [max(0, i - mn - r + 1), min(m, i + mx)).
// One block per series; minima over power-of-two windows by doubling.
__global__ void __launch_bounds__(256)
envelope_kernel(const ElasticJob J, const float *yf, int64_t ys, float2 *env) {
    extern __shared__ float sm[];
    const Band B(J, 16);
    const int m = B.m, n = B.n;
    float *lo0 = sm, *hi0 = sm + m, *lo1 = sm + 2 * m, *hi1 = sm + 3 * m;
    const int full = imin(B.width, m);
    const int lev = 31 - __clz(full);  // 2^lev <= full
    for (int64_t j = blockIdx.x; j < J.cols.count; j += gridDim.x) {
        const float *y = yf + j * ys;
        __syncthreads();
        for (int c = threadIdx.x; c < m; c += 256) lo0[c] = hi0[c] = y[c];
        __syncthreads();
        float *a = lo0, *b = hi0, *a2 = lo1, *b2 = hi1;
        for (int p = 0; p < lev; p++) {
            // window 2^(p + 1) from c (cut at the end, where it is not used)
            for (int c = threadIdx.x; c < m; c += 256) {
                const int d = imin(c + (1 << p), m - 1);
                a2[c] = fminf(a[c], a[d]);
                b2[c] = fmaxf(b[c], b[d]);
            }
            __syncthreads();
            float *t = a; a = a2; a2 = t;
            t = b; b = b2; b2 = t;
        }
        for (int i = threadIdx.x; i < n; i += 256) {
            const int c0 = imax(0, i - B.mn - B.r + 1), c1 = imin(m, i + B.mx);
            float l = WB_FLT_INF, u = -WB_FLT_INF;
            if (c1 - c0 >= (1 << lev)) {
                const int e = c1 - (1 << lev);
                l = fminf(a[c0], a[e]);
                u = fmaxf(b[c0], b[e]);
            } else {  // the band's ends, narrower than the window
                for (int c = c0; c < c1; c++) {
                    l = fminf(l, y[c]);
                    u = fmaxf(u, y[c]);
                }
            }
            env[j * n + i] = make_float2(l, u);
        }
    }
}

// xt[i][q] = x_q[i], rows of `ld` floats
__global__ void __launch_bounds__(256)
transpose_kernel(const float *xf, int64_t xs, int64_t nq, int n, float *xt, int64_t ld) {
    __shared__ float tile[32][33];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int64_t q0 = (int64_t)blockIdx.x * 32;
    const int i0 = blockIdx.y * 32;
    for (int k = ty; k < 32; k += 8)
        tile[k][tx] = (q0 + k < nq && i0 + tx < n) ? xf[(q0 + k) * xs + 3 + i0 + tx] : 0.0f;
    __syncthreads();
    for (int k = ty; k < 32; k += 8)
        if (i0 + k < n && q0 + tx < ld) xt[(int64_t)(i0 + k) * ld + q0 + tx] = tile[tx][k];
}

struct FilterArgs {
    GuidedArgs G;
    EaChunk C;             // the chunk, with the k-th distances
    const float *xt = nullptr;
    int64_t xt_ld = 0;
    const float2 *env = nullptr;  // null: the first filter reads the lower bounds only
    uint32_t *out_items = nullptr;
    unsigned *out_n = nullptr;
    const uint32_t *in_items = nullptr;
    const unsigned *in_n = nullptr;
    unsigned *queue = nullptr;
    float *ring = nullptr;  // [group of 4 columns][thread] float4 rows
    int64_t nth = 0;
};

// bound of a float sum for the pair (file header); +inf while the heap fills
__device__ __forceinline__ float sum_bound(const FilterArgs &F, double scale, int64_t q,
                                           int64_t j, float K, bool penalties) {
    const double d = F.C.cur_dist[q];
    if (!(d < WB_DBL_MAX)) return WB_FLT_INF;
    const float e = __fmaf_ru(6.0e-8f, __fadd_ru(F.G.xr[q].mag, F.G.yr[j].mag), 1e-37f);
    const float root = __fmaf_ru(e, __fsqrt_ru(K), __double2float_ru(d * scale));
    const float g = __fmul_ru(__fmaf_ru(penalties ? 2.0f : 1.0f, K, 16.0f), 6.3e-8f);
    return __fadd_ru(__fmul_ru(__fmul_ru(root, root), __fadd_ru(1.000002f, g)), 1e-30f);
}

__device__ __forceinline__ void append(const FilterArgs &F, bool keep, uint32_t item) {
    const unsigned mask = __ballot_sync(0xffffffffu, keep);
    if (mask == 0) return;
    const int lane = threadIdx.x & 31;
    unsigned base = 0;
    if (lane == 0) base = atomicAdd(F.out_n, __popc(mask));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (keep) F.out_items[base + __popc(mask & ((1u << lane) - 1u))] = item;
}

__global__ void __launch_bounds__(128) lb_filter_kernel(const FilterArgs F) {
    const EaChunk &C = F.C;
    const ElasticJob &J = F.G.J;
    const int64_t q = (int64_t)blockIdx.x * 128 + threadIdx.x;
    const bool mine = q < C.nq;
    const int64_t qq = mine ? q : C.nq - 1;
    double centre = 0.0, scale = 1.0;
    const bool finite = centre_scale(F.G.prep, centre, scale);
    const float K = (float)(J.rows.len + J.cols.len);
    const int n = J.rows.len;
    for (int64_t c0 = (int64_t)blockIdx.y * kLbCols; c0 < C.nc;
         c0 += (int64_t)gridDim.y * kLbCols) {
        float bound[kLbCols], sum[kLbCols];
        const float2 *env[kLbCols];
        bool alive = false;
#pragma unroll
        for (int t = 0; t < kLbCols; t++) {
            const int64_t j = C.j0 + c0 + t;
            bound[t] = -1.0f;
            sum[t] = 0.0f;
            env[t] = F.env + (c0 + t < C.nc ? j : C.j0) * n;
            if (mine && c0 + t < C.nc) {
                bound[t] = sum_bound(F, scale, q, j, K, J.kind == K_ADTW);
                if (C.lower_bound && C.lower_bound[q * C.ny + j] >= C.cur_dist[q]) bound[t] = -1.0f;
                alive |= bound[t] >= 0.0f;
            }
        }
        if (F.env && finite) {
            for (int i0 = 0; i0 < n; i0 += 32) {
                if (!__any_sync(0xffffffffu, alive)) break;
                const int i1 = imin(n, i0 + 32);
#pragma unroll 4
                for (int i = i0; i < i1; i++) {
                    const float x = F.xt[(int64_t)i * F.xt_ld + qq];
#pragma unroll
                    for (int t = 0; t < kLbCols; t++) {
                        const float2 e = __ldg(env[t] + i);
                        const float d = fmaxf(fmaxf(__fsub_rn(x, e.y), __fsub_rn(e.x, x)), 0.0f);
                        sum[t] = __fmaf_rn(d, d, sum[t]);
                    }
                }
                alive = false;
#pragma unroll
                for (int t = 0; t < kLbCols; t++) alive |= sum[t] <= bound[t];
            }
        }
#pragma unroll
        for (int t = 0; t < kLbCols; t++) {
            const bool in = mine && c0 + t < C.nc;
            const bool keep = in && !(sum[t] > bound[t]);
            if (in && !keep) J.out[q * C.ny + C.j0 + c0 + t] = WB_DBL_INF;
            append(F, keep, (uint32_t)((c0 + t) * C.nq + q));
        }
    }
}

// smallest predecessor (with the move's penalty) plus the cost
template <int KIND>
__device__ __forceinline__ float filter_cell(float d, float w, float dg, float up, float lf,
                                             float pen) {
    float best;
    if constexpr (KIND == K_ADTW) best = fminf(__fadd_rn(fminf(up, lf), pen), dg);
    else asm("min.f32 %0, %1, %2, %3;" : "=f"(best) : "f"(dg), "f"(up), "f"(lf));
    if constexpr (KIND == K_WDTW) return __fmaf_rn(__fmul_rn(d, d), w, best);
    else return __fmaf_rn(d, d, best);
}

constexpr int kSweepRows = 16;

template <int KIND, bool MASK>
__device__ __forceinline__ void filter_column(const float (&Pin)[kSweepRows],
                                              float (&Pout)[kSweepRows], float bup, float bdiag,
                                              const float (&x)[kSweepRows], float y,
                                              const float *wq, float pen, unsigned M) {
#pragma unroll
    for (int i = 0; i < kSweepRows; i++) {
        const float dg = i == 0 ? bdiag : Pin[i > 0 ? i - 1 : 0];
        const float up = i == 0 ? bup : Pout[i > 0 ? i - 1 : 0];
        const float w = KIND == K_WDTW ? wq[kSweepRows - 1 - i] : 1.0f;
        float v = filter_cell<KIND>(__fsub_rn(x[i], y), w, dg, up, Pin[i], pen);
        if (MASK) v = ((M >> i) & 1u) ? v : WB_FLT_INF;
        Pout[i] = v;
    }
}

// One thread per pair of the list: strips of 16 rows, the row above a strip in
// a per-thread ring; a warp ends when all its pairs are dropped.
template <int KIND>
__global__ void __launch_bounds__(128) sweep_filter_kernel(const FilterArgs F) {
    constexpr int S = kSweepRows;
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const EaChunk &C = F.C;
    const GuidedArgs &A = F.G;
    const ElasticJob &J = A.J;
    const Band B(J, S);
    const int64_t nth = F.nth;
    float4 *ring = reinterpret_cast<float4 *>(F.ring) + (int64_t)blockIdx.x * 128 + threadIdx.x;
    double centre = 0.0, scale = 1.0;
    const bool finite = centre_scale(A.prep, centre, scale);
    const float pen = KIND == K_ADTW ? __double2float_rd(J.p * scale * scale) : 0.0f;
    const float K = (float)(B.n + B.m);
    const int64_t n_in = *F.in_n;
    const float4 INF4 = make_float4(WB_FLT_INF, WB_FLT_INF, WB_FLT_INF, WB_FLT_INF);
    for (;;) {
        unsigned t = 0;
        if (lane == 0) t = atomicAdd(F.queue, 1u);
        const int64_t at = (int64_t)__shfl_sync(FULL, t, 0) * 32 + lane;
        if (at - lane >= n_in) break;
        const bool active = at < n_in;
        const uint32_t item = F.in_items[active ? at : n_in - 1];
        const int64_t q = item % C.nq, j = C.j0 + item / C.nq;
        const float *xr = A.xf + q * A.xs + 3;
        const float *yr = A.yf + j * A.ys;
        const float bound = sum_bound(F, scale, q, j, K, KIND == K_ADTW);
        bool alive = active;
        float result = 0.0f;
        if (finite) {
            // row 0
            const int lim = imin(B.m, B.mx);
            const float x0 = xr[0];
            float acc = 0.0f;
            for (int g = 0; g <= (lim - 1) >> 2; g++) {
                const float4 y = reinterpret_cast<const float4 *>(yr)[g];
                const float yq[4] = {y.x, y.y, y.z, y.w};
                float v[4];
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const int c = 4 * g + k;
                    const float d = __fsub_rn(x0, yq[k]);
                    const float sq = __fmul_rn(d, d);
                    acc = KIND == K_WDTW ? __fmaf_rn(sq, A.wext[A.woff + imax(c - 1, 0)], acc)
                                         : __fadd_rn(sq, acc);
                    v[k] = c < lim ? acc : WB_FLT_INF;
                }
                ring[(int64_t)g * nth] = make_float4(v[0], v[1], v[2], v[3]);
            }
            int pg0 = 0, pg1 = (lim - 1) >> 2;
            for (int s = 0; s < B.ns; s++) {
                const int i0 = 1 + s * S, rows = imin(S, B.n - i0);
                const int cs = B.cs(s, S), ce = B.ce(s, S);
                const int g0 = cs >> 2, g1 = (ce - 1) >> 2;
                int bstart = 0x7fffffff, bend = 0;
                if (rows == S) {
                    bstart = imax(cs, i0 + S - 1 + B.lo);
                    bend = imin(s == B.ns - 1 ? imin(ce, (B.m - 1) & ~3) : ce, i0 + B.mx);
                }
                float x[S], P[S], Q[S];
                float low = WB_FLT_INF;  // smallest value of the strip's bottom row
#pragma unroll
                for (int k = 0; k < S; k++) {
                    x[k] = i0 + k < B.n ? xr[i0 + k] : WB_FLT_INF;
                    P[k] = WB_FLT_INF;
                }
                auto up4 = [&](int g) {
                    return g >= pg0 && g <= pg1 ? ring[(int64_t)g * nth] : INF4;
                };
                float bd = up4(g0 - 1).w;
                float4 nu = up4(g0), nnu = up4(g0 + 1);
                const float4 *y4 = reinterpret_cast<const float4 *>(yr);
                float4 ny = y4[g0];
                for (int g = g0; g <= g1; g++) {
                    const float4 u = nu, y = ny;
                    nu = nnu;
                    nnu = up4(g + 2);
                    if (g < g1) ny = y4[g + 1];
                    float w[S + 4];
                    if constexpr (KIND == K_WDTW) {
                        const float4 *w4 = reinterpret_cast<const float4 *>(
                            A.wext + (A.woff + 4 * g - i0 - (S - 1)));
#pragma unroll
                        for (int k = 0; k < S / 4 + 1; k++) {
                            const float4 t4 = w4[k];
                            w[4 * k] = t4.x;
                            w[4 * k + 1] = t4.y;
                            w[4 * k + 2] = t4.z;
                            w[4 * k + 3] = t4.w;
                        }
                    }
                    float4 o;
                    if (4 * g >= bstart && 4 * g + 3 < bend) {
                        filter_column<KIND, false>(P, Q, u.x, bd, x, y.x, w, pen, 0u);
                        o.x = Q[S - 1];
                        filter_column<KIND, false>(Q, P, u.y, u.x, x, y.y, w + 1, pen, 0u);
                        o.y = P[S - 1];
                        filter_column<KIND, false>(P, Q, u.z, u.y, x, y.z, w + 2, pen, 0u);
                        o.z = Q[S - 1];
                        filter_column<KIND, false>(Q, P, u.w, u.z, x, y.w, w + 3, pen, 0u);
                        o.w = P[S - 1];
                    } else {
                        const int e = 4 * g - i0 - B.lo;
                        auto masked = [&](int k, const float(&Pin)[S], float(&Pout)[S],
                                          float bup, float bdg, float yk) {
                            const unsigned M = 4 * g + k < B.m ? band_rows(e + k, B.width) : 0u;
                            filter_column<KIND, true>(Pin, Pout, bup, bdg, x, yk, w + k, pen, M);
                            if (s == B.ns - 1 && 4 * g + k == B.m - 1) {
#pragma unroll
                                for (int h = 0; h < S; h++)
                                    if (h < rows) result = Pout[h];
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
                    low = fminf(low, fminf(fminf(o.x, o.y), fminf(o.z, o.w)));
                    bd = u.w;
                    ring[(int64_t)g * nth] = o;
                }
                pg0 = g0;
                pg1 = g1;
                if (s < B.ns - 1) {
                    alive = alive && !(low > bound);
                    if (!__any_sync(FULL, alive)) break;
                }
            }
        }
        const bool keep = alive && !(result > bound);
        if (active && !keep) J.out[q * C.ny + j] = WB_DBL_INF;
        append(F, keep, item);
    }
}

// Each chunk ends with a guided evaluation of few pairs, whose latency (about
// 2 ms at length 512) favours few chunks, while a chunk lets through k kGrowth
// candidates per query: growth 4, 8, 16 and 64 took 12.5, 10.5, 11.0 and
// 14.5 ms for the shape of the file header.
constexpr int64_t kGrowth = 8;

}  // namespace

struct GuidedArgmin::Impl {
    GuidedContext ctx;
    FilterArgs F;
    int sweep_grid = 0;
    unsigned *counters = nullptr;  // per chunk: items of both lists, queue
};

constexpr int kMaxChunks = 40;

// (the pairs of a batch are below 2^31, so an item fits 32 bits)
bool argmin_guided_supported(const ElasticJob &J) {
    if (J.kind != K_DTW && J.kind != K_WDTW && !(J.kind == K_ADTW && J.p >= 0.0)) return false;
    if (J.mode != PM_ALL || J.all_zero) return false;
    if (J.rows.count * J.cols.count >= (int64_t)1 << 31) return false;
    if (getenv("WB_GPU_ARGMIN") || getenv("WB_GPU_ARGMIN_FORM")) return false;
    return guided_list_bytes(J, 1) > 0;
}

// pairs resident in the guided kernel: two blocks per SM, since the chunks
// after the first hold few pairs
static int64_t argmin_guided_pairs(const ElasticJob &J) {
    return std::min<int64_t>(J.rows.count * J.cols.count,
                             (int64_t)2 * device_info().sm_count * 128);
}

static int sweep_blocks(const ElasticJob &J) {
    int nb = 0;
    switch (J.kind) {
        case K_DTW:
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, sweep_filter_kernel<K_DTW>, 128, 0);
            break;
        case K_WDTW:
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, sweep_filter_kernel<K_WDTW>, 128, 0);
            break;
        default:
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, sweep_filter_kernel<K_ADTW>, 128, 0);
    }
    return imax(nb, 1) * device_info().sm_count;
}

std::vector<int64_t> argmin_guided_chunks(int64_t nq, int64_t ny, int64_t k) {
    // the first chunk runs without bounds: enough candidates for the heap and,
    // with few queries, for the SMs
    const int64_t warm = (int64_t)device_info().sm_count * 64 / std::max<int64_t>(nq, 1);
    std::vector<int64_t> at{0};
    int64_t c = std::max<int64_t>({4 * k, 32, warm});
    while (at.back() < ny) {
        at.push_back(std::min(ny, at.back() + c));
        c *= kGrowth;
    }
    return at;
}

static bool has_envelope(const ElasticJob &J) {
    return J.kind != K_WDTW && J.cols.len <= kLbMaxLen;
}

size_t argmin_guided_bytes(const ElasticJob &J) {
    const int64_t pairs = J.rows.count * J.cols.count;
    const int64_t ld = (J.rows.count + 31) / 32 * 32;
    size_t b = guided_list_bytes(J, argmin_guided_pairs(J)) + 2 * align256(pairs * 4) +
               align256(3 * kMaxChunks * sizeof(unsigned)) +
               align256((size_t)sweep_blocks(J) * 128 * ((J.cols.len + 3) / 4 + 1) * 16) + 8192;
    if (has_envelope(J))
        b += align256((size_t)ld * J.rows.len * 4) +
             align256((size_t)J.cols.count * J.rows.len * 8);
    return b;
}

// Prepares the batch J (rows = its queries); false when the workspace left
// beyond `leave` is too small.
int GuidedArgmin::prepare(const ElasticJob &J, Workspace &ws, size_t leave, bool &ok) {
    ok = false;
    if (ws.remaining() < leave + argmin_guided_bytes(J)) return WB_OK;
    cudaStream_t s = ws.stream();
    impl_ = std::make_shared<Impl>();
    FilterArgs &F = impl_->F;
    const int64_t pairs = J.rows.count * J.cols.count;
    WB_TAKE(list1, uint32_t, ws, pairs);
    WB_TAKE(list2, uint32_t, ws, pairs);
    WB_TAKE(counters, unsigned, ws, 3 * kMaxChunks);
    impl_->sweep_grid = sweep_blocks(J);
    F.nth = (int64_t)impl_->sweep_grid * 128;
    WB_TAKE(ring, float, ws, (size_t)F.nth * ((J.cols.len + 3) / 4 + 1) * 4);
    F.ring = ring;
    impl_->counters = counters;
    F.out_items = list1;
    F.in_items = list2;  // the two lists; launch_chunk assigns their roles
    float *xt = nullptr;
    float2 *env = nullptr;
    const int64_t ld = (J.rows.count + 31) / 32 * 32;
    if (has_envelope(J)) {
        xt = ws.take<float>((size_t)ld * J.rows.len);
        env = ws.take<float2>((size_t)J.cols.count * J.rows.len);
        if (!xt || !env) return fail(WB_ENOMEM, "workspace reservation exceeded");
    }
    WB_TRY(guided_prepare(J, ws, leave, argmin_guided_pairs(J), impl_->ctx));
    if (!impl_->ctx.args.prep) return WB_OK;
    const GuidedArgs &A = impl_->ctx.args;
    F.G = A;
    F.xt = xt;
    F.xt_ld = ld;
    F.env = env;
    WB_CUDA(cudaMemsetAsync(counters, 0, 3 * kMaxChunks * sizeof(unsigned), s));
    if (env) {
        const dim3 tg((unsigned)((J.rows.count + 31) / 32), (unsigned)((J.rows.len + 31) / 32));
        transpose_kernel<<<tg, 256, 0, s>>>(A.xf, A.xs, J.rows.count, J.rows.len, xt, ld);
        WB_LAUNCH_CHECK("transpose_kernel");
        const size_t smem = (size_t)4 * J.cols.len * sizeof(float);
        WB_CUDA(allow_shared(envelope_kernel, smem));
        const int64_t cap = (int64_t)device_info().sm_count * 8;
        envelope_kernel<<<(int)std::min(cap, J.cols.count), 256, smem, s>>>(J, A.yf, A.ys, env);
        WB_LAUNCH_CHECK("envelope_kernel");
    }
    ok = true;
    return WB_OK;
}

// Distances of the candidates of chunk number `index`: exact where the
// reference could push the candidate, else +inf; the pairs left to the full
// recurrence hold kGuidedPending.
int GuidedArgmin::launch_chunk(int index, const EaChunk &C, cudaStream_t s,
                               ElasticJob &second) {
    if (index >= kMaxChunks) return fail(WB_EINVAL, "too many candidate chunks");
    GuidedContext ctx = impl_->ctx;
    const ElasticJob &J = ctx.args.J;
    ctx.args.col0 = C.j0;
    if (index == 0) {
        ctx.args.n_all = C.nq * C.nc;
    } else {
        FilterArgs F = impl_->F;
        uint32_t *l1 = F.out_items, *l2 = const_cast<uint32_t *>(F.in_items);
        unsigned *n1 = impl_->counters + 3 * index, *n2 = n1 + 1, *queue = n1 + 2;
        F.C = C;
        F.out_items = l1;
        F.out_n = n1;
        const int64_t groups = (C.nc + kLbCols - 1) / kLbCols;
        const dim3 grid((unsigned)((C.nq + 127) / 128),
                        (unsigned)std::min<int64_t>(groups, 65535));
        lb_filter_kernel<<<grid, 128, 0, s>>>(F);
        WB_LAUNCH_CHECK("lb_filter_kernel");
        F.in_items = l1;
        F.in_n = n1;
        F.out_items = l2;
        F.out_n = n2;
        F.queue = queue;
        const int sg = (int)std::min<int64_t>(impl_->sweep_grid, (C.nq * C.nc + 127) / 128);
        switch (J.kind) {
            case K_DTW: sweep_filter_kernel<K_DTW><<<sg, 128, 0, s>>>(F); break;
            case K_WDTW: sweep_filter_kernel<K_WDTW><<<sg, 128, 0, s>>>(F); break;
            default: sweep_filter_kernel<K_ADTW><<<sg, 128, 0, s>>>(F); break;
        }
        WB_LAUNCH_CHECK("sweep_filter_kernel");
        ctx.args.items = l2;
        ctx.args.n_items = n2;
    }
    WB_TRY(guided_run(ctx, s));
    second.pending = &ctx.args.prep->pending;
    second.tail_cap = ctx.args.tail_cap;
    return WB_OK;
}

}  // namespace wb
