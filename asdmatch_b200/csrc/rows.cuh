// Embedding rows (EMBED mode) as packed keys: a row's candidate indices, one
// field per query vertex, in as few 64-bit words as hold them.  Candidate
// sets are ascending, so the order of the keys (word 0 first) is the
// lexicographic order of the rows' vertex ids.
#pragma once

#include "cs.cuh"

namespace asdm {

struct RowLayout {
    uint32_t words = 0;
    std::vector<uint32_t> word, shift, bits;  // by query vertex
    std::vector<uint32_t> word_bits;          // used bits of each word (the low ones)
};

RowLayout row_layout(const asdm_cs &cs);

// The rows of `keys` (word k of row r at keys[k * cap + r]) in ascending
// order, as vertex ids, into the host array out (rows x n).
int sorted_rows(const asdm_cs &cs, const RowLayout &lay, const unsigned long long *keys, uint64_t cap, uint64_t rows,
                uint32_t *out);

}  // namespace asdm
