// The order of a tile's steps over its K chunks: fetches run kStages - 1 chunks
// ahead of the products, a stage is refilled only once the products that read
// it are complete, and whatever happens the return comes after a wait for the
// last products issued.  Device code for the kernel, host code for its test.
#pragma once

#ifdef __CUDACC__
#define ASDM_STEPS __device__ __forceinline__
#else
#define ASDM_STEPS inline
#endif

namespace asdm {
namespace tc {

// fetch(i): starts chunk i's copy into stage i % kStages (nothing past the
// last chunk).  issue(i): waits for chunk i's copy and issues its products.
// wait(i): a bounded wait for chunk i's products and all before them; false
// when it ran out.  all(x): whether every thread of the block has x.  Returns
// whether every wait was met; when one ran out, no more products are issued and
// those in flight get one more wait, the last chunk's, which covers them all:
// the caller then releases the accumulator that they write.
template <int kStages, typename Fetch, typename Issue, typename Wait, typename All>
ASDM_STEPS bool run_chunks(int nc, Fetch fetch, Issue issue, Wait wait, All all) {
#pragma unroll
    for (int i = 0; i < kStages - 1; ++i) fetch(i);
    bool ok = true;
    int i = 0;
    for (; i < nc && ok; ++i) {
        issue(i);
        // the next fetch goes into the stage that chunk i - 1 was read from
        ok = all(i == 0 || wait(i - 1));
        if (ok) fetch(i + kStages - 1);
    }
    if (i > 0) {
        const bool last = wait(i - 1);
        ok = all(ok && last);
    }
    return ok;
}

}  // namespace tc
}  // namespace asdm
