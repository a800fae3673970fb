// The wait of an idle warp for a record in its mailbox.  Device code for the
// enumeration kernels, host code for its test.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define ASDM_IDLE __device__ __forceinline__
#else
#define ASDM_IDLE inline
#endif

namespace asdm {

enum : uint32_t { kMailEmpty = 0, kMailRecord = 1, kMailDone = 2 };
constexpr uint64_t kHandoffNs = 1000000000ull;  // longest wait for a record once claimed
constexpr uint32_t kIdleCheck = 256;            // polls between looks at the clock and the stop flags

// Returns whether the mailbox holds a record.  io.ended(): the run ended before
// the mailbox was emptied; io.mail(): its flag; io.stopped(): a stop flag of
// the run; io.take_back(): takes this warp off the idle warps, false when a
// donor has claimed it already; io.lost(): marks the run as not to be trusted.
//
// The wait ends with a record, the end mail, a stop flag or the time `until`.
// In the last two a claimed warp waits for its record, kHandoffNs at most: its
// donor has counted it as working.  Should that record not come (it cannot by
// the donor's code), the count of working warps stays above zero and no end
// mail follows, so the other idle warps leave by the stop flag that lost() sets.
template <typename Io>
ASDM_IDLE bool idle_wait(Io &io, uint64_t until) {
    bool claimed = false;
    if (io.ended()) return false;
    for (uint32_t it = 0;; ++it) {
        const uint32_t f = io.mail();
        if (f != kMailEmpty) return f == kMailRecord;
        if ((it & (kIdleCheck - 1)) == kIdleCheck - 1 && ((!claimed && io.stopped()) || io.now() > until)) {
            if (claimed) {
                io.lost();
                return false;
            }
            if (io.take_back()) return false;
            claimed = true;
            until = io.now() + kHandoffNs;
        }
        io.nap();
    }
}

}  // namespace asdm
