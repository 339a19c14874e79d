// argmin.cu -- k-nearest-neighbour selection with the reference's heap.
//
// The distance kernel has produced, for every (query i, candidate j), the
// distance the metric's eadistance returns when it does not abandon, and the
// abandon key K(i, j): the largest per-row minimum of the recurrence.  The
// reference abandons a pair iff some checked row's minimum exceeds the
// threshold, i.e. iff K(i, j) > threshold.  Replaying _ArgMinBatch.__call__
// (distance/_cdistance.pyx:1302-1345) over j in order with those two numbers
// reproduces its pushes, its heap (utils/_misc.pyx:18-107) and therefore its
// output order exactly, including for metrics whose abandoning is not
// monotone (negative adtw penalty, band-edge zeros of lcss/edr/erp/msm/twe).

#include "argmin.cuh"

namespace wb {

// One warp per query.  The k-th distance never increases, so of 32 candidates
// only those below its value before them can be pushed; the warp finds these
// at once and goes through them in order, with the reference's tests against
// the heap's current k-th distance (a thread per query, walking its candidates
// alone with uncoalesced reads, took 1.1 ms for 500 queries x 2000 candidates;
// this takes 0.1 ms).
__global__ void __launch_bounds__(128) argmin_replay_kernel(const ArgminJob J) {
    const double INF = __longlong_as_double(0x7ff0000000000000LL);
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t i = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < J.nx;
         i += warps) {
        int64_t *hi = J.heap_idx + i * J.k;
        double *hv = J.heap_val + i * J.k;
        const double *drow = J.dist + i * J.ny;
        const double *krow = J.key ? J.key + i * J.ny : nullptr;
        const double *lb = J.lower_bound ? J.lower_bound + i * J.ny : nullptr;
        double distance = INF;
        int64_t n = 0;
        if (J.resume) {
            n = J.state_n[i];
            distance = J.state_dist[i];
        }
        const int64_t j1 = J.j1 < 0 ? J.ny : J.j1;
        if (!J.never_push) {
            for (int64_t jb = J.j0; jb < j1; jb += 32) {
                const int64_t j = jb + lane;
                double d = INF, l = -INF;
                if (j < j1) {
                    d = drow[j];
                    if (lb) l = lb[j];
                }
                unsigned todo = __ballot_sync(FULL, j < j1 && !(l >= distance) && d < distance);
                while (todo) {
                    const int t = __ffs(todo) - 1;
                    todo &= todo - 1;
                    const double dt = __shfl_sync(FULL, d, t);
                    const double lt = __shfl_sync(FULL, l, t);
                    if (lane == 0 && !(lt >= distance) && dt < distance) {
                        // abandoned: eadistance returns inf
                        const bool gone =
                            krow && krow[jb + t] >
                                        abandon_threshold(J.metric, distance, J.xl, J.yl);
                        if (!gone) {
                            heap_push(hi, hv, n, J.k, jb + t, dt);
                            distance = (n == J.k) ? hv[0] : INF;
                        }
                    }
                    distance = __shfl_sync(FULL, distance, 0);
                }
            }
        }
        if (lane == 0) {
            if (J.state_n) {
                J.state_n[i] = n;
                J.state_dist[i] = distance;
            }
            if (J.finish) {
                for (int64_t t = 0; t < J.k; t++) {
                    J.out_idx[i * J.k + t] = t < n ? hi[t] : 0;
                    J.out_dist[i * J.k + t] = t < n ? hv[t] : 0.0;
                }
            }
        }
    }
}

int launch_argmin_replay(const ArgminJob &J, cudaStream_t s) {
    if (J.nx == 0) return WB_OK;
    const int64_t cap = (int64_t)device_info().sm_count * 16;
    const int64_t g = (J.nx + 3) / 4;
    argmin_replay_kernel<<<(int)(g < cap ? g : cap), 128, 0, s>>>(J);
    WB_LAUNCH_CHECK("argmin_replay_kernel");
    return WB_OK;
}

}  // namespace wb
