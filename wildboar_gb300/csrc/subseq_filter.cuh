// subseq_filter.cuh -- float32 window filter of the dtw subsequence minimum
// (subseq_filter.cu).
#pragma once

#include "elastic.cuh"

namespace wb {

// The filter takes the job (max_band: its widest half-band); `total` packed
// shapelet values.
bool subseq_filter_supported(const SubseqElasticJob &J, int kind, int max_band, int64_t total);
size_t subseq_filter_bytes(const SubseqElasticJob &J, int64_t total);
// Writes the results of the pairs it settles and sets J.kept / J.redo, so that
// launch_elastic_subseq(J) scans the others.  gring, P, grid: that kernel's.
int launch_subseq_filter(SubseqElasticJob &J, int64_t total, double *gring, int P, int grid,
                         Workspace &ws, cudaStream_t s);

}  // namespace wb
