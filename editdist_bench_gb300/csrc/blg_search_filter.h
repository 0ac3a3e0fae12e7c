// The tensor-core filter of thresholded searches (blg_search_filter.cu).
#pragma once
#include <cuda_runtime.h>

#include "blg_internal.h"

namespace blg {

constexpr int kFltMaxTiles = 512;    // tiles of 128 queries in a launch

// Pairs the filter lets through: (place of the query among the sequential
// queries by length) << 32 | sorted choice; count may pass cap (the list ran
// full). count[0], and count[1], the fill items claimed, are zero before the
// filter.
struct PasserList {
    unsigned long long *item;
    unsigned long long *count;
    unsigned long long cap;
};

// What the repair launch (k_search_band in place) needs where a list ran full:
// its survivor plan's inputs, and the gate that lets it run (count past cap).
struct RepairPlan {
    const int64_t *lstart;
    int64_t min_len, n_len;
    int jobsz;
    ResultList gate;
};

// fill: the output to set to k + 1 (n = 0: none); whole_fill: by the filter
// alone, else the solver goes on with it. folded: signatures of half the bins.
// wait_polls: the roles' waits on one another give up after that many polls (-1:
// the normal bound); a run that did raises ST_QUEUE_TIMEOUT.
cudaError_t launch_filter_pairs(cudaStream_t st, int sms, const SurvClasses &C, int nq, const uint32_t *qsig,
                                const uint32_t *csig, bool folded, const int64_t *lstart, int64_t min_len,
                                int64_t n_len, int k, const PasserList &L, const BatchFill &fill, bool whole_fill,
                                int32_t wait_polls, uint32_t *status);
// Results <= k into `out` (L.item null) or into L. longest: of the queries.
cudaError_t launch_solve_passers(cudaStream_t st, int sms, const SurvClasses &C, const DevStrings &Q,
                                 const DevStrings &CS, const int32_t *perm, const uint4 *ccnt, const uint4 *qcnt,
                                 int64_t longest, int k, int dtype, void *out, int64_t nc, const PasserList &P,
                                 const ResultList &L, const BatchFill &fill, const RepairPlan &plan, uint32_t *status);
// L's results into the output; a list that ran full: the fill, the plan and
// the gate of the repair launch.
cudaError_t launch_solve_finish(cudaStream_t st, int sms, const SurvClasses &C, int k, const PasserList &P,
                                const ResultList &L, const BatchFill &fill, const RepairPlan &plan);

}  // namespace blg
