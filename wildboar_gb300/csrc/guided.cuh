// guided.cuh -- FP64 distances on the cells a 32-bit sweep cannot rule out
// (guided.cu).
#pragma once

#include <algorithm>
#include <cstring>

#include "elastic.cuh"

namespace wb {

// Output of a pair left to the full recurrence (a NaN payload no arithmetic
// produces).
constexpr long long kGuidedPending = 0x7ff8d7a05e1e57edLL;

struct GuidedPrep {
    long long lo, hi;            // order codes of the smallest / largest input
    unsigned long long queue;    // next tile of 32 pairs
    unsigned long long pending;  // pairs left to the full recurrence
};

// Extremes of a series: fixed point, and the largest float magnitude.
struct GuidedRange {
    int lo, hi;
    float mag;
};

struct GuidedArgs {
    ElasticJob J;
    const float *xf = nullptr, *yf = nullptr;  // centred, scaled, padded float series
    const int *xq = nullptr, *yq = nullptr;    // the same in fixed point
    int64_t xs = 0, ys = 0;                    // their strides
    const GuidedRange *xr = nullptr, *yr = nullptr;
    const float *wext = nullptr;  // wdtw: weight of i - j at woff + (j - i)
    int woff = 0;
    GuidedPrep *prep = nullptr;
    // per resident thread, interleaved [...][thread]
    int64_t nth = 0;
    uint4 *ckrow = nullptr;   // [strip + 1][group of 4 columns] bottom rows
    uint4 *ckcol = nullptr;   // [strip][block][S / 4] last columns of the blocks
    uint32_t *list = nullptr;  // [entry][word] collected blocks
    double *brow = nullptr;    // [2][column] FP64 bottom rows of two strips
    int groups = 0, blocks = 0, list_cap = 0, brow_cols = 0;
};

// Evaluates the job on what is left of the workspace beyond `leave` bytes;
// *pending is null when
// the job is not guided (or too little is left), else the device counter of
// the pairs whose output is kGuidedPending.
int launch_guided(const ElasticJob &job, Workspace &ws, size_t leave,
                  unsigned long long **pending);

#ifdef __CUDACC__
__device__ __forceinline__ bool is_pending(double v) {
    return __double_as_longlong(v) == kGuidedPending;
}
#endif

}  // namespace wb
