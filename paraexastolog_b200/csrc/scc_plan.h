// Host rules of the SCC-resident solver (k_sw_scc in sweep.cu): sizes and launch shapes,
// without CUDA types, so that they can be checked on a machine without a GPU.
#pragma once

#include <algorithm>
#include <cstdint>

namespace esl {

// Group-sized vectors that k_sw_scc keeps in memory, in the order of SccArgs::own.  The
// first five are per odd row (kSccBig); kSccGrid uses all of them.
enum SccOwn { kOwnR0, kOwnD, kOwnDS, kOwnQ, kOwnBS, kOwnA, kOwnW, kOwnR, kOwnV, kOwnP, kOwnT, kOwnIQ, kOwnCount };

// Rows of vector j in a group of `even` and `odd` rows.  kOwnA holds odd rows while an
// operator is applied to it, and 1 / q of the even rows before that.
inline uint32_t scc_own_rows(int j, uint32_t even, uint32_t odd) {
    const uint32_t rows = j == kOwnW || j == kOwnIQ ? even : j == kOwnA ? std::max(even, odd) : odd;
    return std::max<uint32_t>(rows, 1);
}

}  // namespace esl
