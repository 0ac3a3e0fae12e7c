// The bit-sliced exact search (blg_search_bits.cu): its launch description.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

#include "blg_internal.h"

namespace blg {

struct BitSearch {
    DevStrings Q;                    // the queries' bytes
    const int32_t *qidx, *qlen;      // the search's queries by length: row and length
    int nq;
    TransposedChoices T;
    const uint16_t *order;           // per tile: its choices' positions, longest first
    uint32_t *scratch;               // deltas between stripes (null: no query is longer than 64)
    int64_t scratch_words;           // per warp (bits_scratch_words)
    int nsym;                        // distinct bytes of the queries, at most 255
    uint8_t map[256];                // byte -> symbol 1..nsym; 0: in no query (rows of symbol nsym + 1: valid queries)
    int groups;                      // of 32 queries
    const int64_t *weight;           // [groups + 1] weight of the units before each group, the longest queries first
    // set by the launcher
    int stride;                      // words between symbols
    int per;                         // units of one group per CTA (small launches); 0: parts of equal weight
};

// Shared-memory table of a launch (bytes), warps of its grid, scratch words
// per warp for choices of at most that length.
size_t bits_table_bytes(int nsym, int64_t longest);
int bits_warps(int sms);
int64_t bits_scratch_words(int64_t longest_choice);
int64_t bits_unit_weight(int64_t longest);
cudaError_t launch_search_bits(cudaStream_t st, int sms, BitSearch B, int64_t longest, int dtype, void *out,
                               uint32_t *status);

}  // namespace blg
