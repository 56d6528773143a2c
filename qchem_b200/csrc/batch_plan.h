// batch_plan.h -- how an ERI batch is cut into groups of 32 lanes (pattern_scan_kernel, fock_kernels.cu).
#pragma once
#include <cuda_runtime.h>

#include "qcg_internal.h"

namespace qcg {

// Buckets (contraction patterns) in visiting order: bucket b's quartets are entries first[b] .. first[b + 1) of the
// batch's order and its groups group[b] .. group[b + 1); 1 << lanes[b] lanes share a quartet.
struct BatchPlanDev
{
    int first[257], group[257], lanes[256];
};

// The sort's bucket counters stand kBucketStride ints apart, each on a line of its own: 250 000 updates of 81 counters
// took 36 or 69 us side by side, as the 1 KiB they shared happened to be aligned, and 13 so.
constexpr int kBucketStride = 32, kBucketInts = 256 * kBucketStride;

// primitive loops up to this length are never split for their length alone
constexpr int kBatchChain = 4;

// counting sort of a quartet batch by contraction pattern -> order (a permutation of 0..nq-1), and the plan for
// `ctas` thread blocks
void launch_pattern_sort(const BasisDev& bs, const int4* quartets, long long nq, unsigned char* key, int* hist,
                         int* cursor, int* order, int ctas, BatchPlanDev* plan, cudaStream_t st, int nsm);

}   // namespace qcg
