// Local-count matrices (|Vg| x n, row-major) on their way to the caller.
//
// A matrix is zero outside the candidates: for 8 queries of 4 and 5 vertices
// on 10^6 vertices, 290 MB hold 1.6 x 10^6 nonzero entries.  Large matrices
// are therefore zeroed by host threads while the device works, and only the
// candidates' entries are gathered, copied and scattered; small ones, and
// ones that are mostly candidates, are copied whole.
#pragma once

#include <atomic>
#include <thread>
#include <utility>

#include "cs.cuh"

namespace asdm {

// Zeroes host buffers with several threads; join() (or the destructor) waits.
class HostFill {
public:
    void start(const std::vector<std::pair<uint64_t *, uint64_t>> &bufs);
    void join();
    bool large() const { return large_; }  // whether the buffers are worth the threads and the gathered read
    ~HostFill() { join(); }

private:
    struct Piece {
        uint64_t *p;
        uint64_t words;
    };
    std::vector<Piece> pieces_;
    std::atomic<size_t> next_{0};
    std::vector<std::thread> threads_;
    bool large_ = false;
    void work();
};

struct LocalRead {
    const asdm_cs *cs;
    const unsigned long long *block;  // device matrix
    uint64_t *host;
};

// Copies the matrices to their host buffers, which `fill` has zeroed (joined
// here) or is zeroing.
int read_locals(asdm_graph *G, const std::vector<LocalRead> &reads, HostFill &fill);

}  // namespace asdm
