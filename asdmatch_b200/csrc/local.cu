#include <algorithm>
#include <system_error>

#include "local.cuh"

namespace asdm {
namespace {

// Buffers of this many bytes in all are filled by threads (starting them costs
// about 0.3 ms, zeroing 8 MB of fresh pages about 2 ms).
constexpr uint64_t kThreadedBytes = 8u << 20;
constexpr uint64_t kPieceWords = 1u << 18;  // 2 MiB
constexpr unsigned kMaxThreads = 16;

unsigned thread_count(uint64_t pieces) {
    const unsigned hw = std::thread::hardware_concurrency();
    return (unsigned)std::min<uint64_t>(pieces, std::min(kMaxThreads, std::max(1u, hw)));
}

// Runs f(k) for k in [0, n) on several threads.
template <typename F>
void parallel_for(size_t n, F f) {
    std::atomic<size_t> next{0};
    auto work = [&]() {
        for (size_t k; (k = next.fetch_add(1)) < n;) f(k);
    };
    std::vector<std::thread> threads;
    const unsigned t = thread_count(n);
    try {
        for (unsigned i = 1; i < t; ++i) threads.emplace_back(work);
    } catch (const std::system_error &) {
        // fewer threads then
    }
    work();
    for (auto &x : threads) x.join();
}

struct GatherSeg {
    const uint32_t *cand;              // C(u)
    const unsigned long long *block;   // |Vg| x n
    uint32_t n, u;
    unsigned long long start;          // first entry of this segment
};

// The candidates' entries of every matrix, side by side, with their vertices.
__global__ void gather_local(const GatherSeg *__restrict__ segs, uint32_t nseg, unsigned long long total,
                             unsigned long long *__restrict__ val, uint32_t *__restrict__ vertex) {
    for (unsigned long long t = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; t < total;
         t += (unsigned long long)gridDim.x * blockDim.x) {
        uint32_t lo = 0, hi = nseg;
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (segs[mid].start <= t) lo = mid; else hi = mid;
        }
        const GatherSeg sg = segs[lo];
        const uint32_t v = sg.cand[t - sg.start];
        val[t] = sg.block[(unsigned long long)v * sg.n + sg.u];
        vertex[t] = v;
    }
}

}  // namespace

void HostFill::work() {
    for (size_t k; (k = next_.fetch_add(1)) < pieces_.size();) std::fill(pieces_[k].p, pieces_[k].p + pieces_[k].words, 0ull);
}

void HostFill::start(const std::vector<std::pair<uint64_t *, uint64_t>> &bufs) {
    uint64_t words = 0;
    for (const auto &b : bufs) words += b.second;
    large_ = words * sizeof(uint64_t) >= kThreadedBytes;
    if (!large_) {
        for (const auto &b : bufs) std::fill(b.first, b.first + b.second, 0ull);
        return;
    }
    for (const auto &b : bufs)
        for (uint64_t w = 0; w < b.second; w += kPieceWords)
            pieces_.push_back(Piece{b.first + w, std::min(kPieceWords, b.second - w)});
    const unsigned t = thread_count(pieces_.size());
    try {
        for (unsigned i = 0; i < t; ++i) threads_.emplace_back(&HostFill::work, this);
    } catch (const std::system_error &) {
        // join() does what no thread did
    }
}

void HostFill::join() {
    if (!pieces_.empty()) work();
    for (auto &t : threads_) t.join();
    threads_.clear();
    pieces_.clear();
}

int read_locals(asdm_graph *G, const std::vector<LocalRead> &reads, HostFill &fill) {
    cudaStream_t s = G->stream;
    std::vector<GatherSeg> segs;
    std::vector<uint64_t *> host;  // by segment
    unsigned long long total = 0;
    std::vector<const LocalRead *> whole;
    for (const LocalRead &r : reads) {
        const asdm_cs &c = *r.cs;
        const uint32_t n = c.q.n;
        uint64_t cands = 0;
        for (uint32_t u = 0; u < n; ++u) cands += c.ncand[u];
        // an entry costs 12 bytes gathered, 8 in the matrix, and a scattered store
        if (!fill.large() || cands * 4 > (uint64_t)G->d.n * n) {
            whole.push_back(&r);
            continue;
        }
        for (uint32_t u = 0; u < n; ++u) {
            segs.push_back(GatherSeg{c.d_cand + c.cand_base[u], r.block, n, u, total});
            host.push_back(r.host);
            total += c.ncand[u];
        }
    }
    GatherSeg *d_segs = nullptr;
    unsigned long long *d_val = nullptr;  // values, then vertices
    const uint64_t words = total + (total + 1) / 2;
    std::vector<unsigned long long> back;
    int rc = ASDM_OK;
    if (total && (rc = dalloc(&d_segs, segs.size(), s)) == ASDM_OK) rc = dalloc(&d_val, words, s);
    if (rc == ASDM_ERR_OOM) {  // no room for the gathered entries: every matrix is copied whole
        clear_error();
        rc = ASDM_OK;
        total = 0;
        whole.clear();
        for (const LocalRead &r : reads) whole.push_back(&r);
    }
    do {
        if (rc != ASDM_OK) break;
        if (total) {
            if (upload_async(G, d_segs, segs.data(), segs.size() * sizeof(GatherSeg)) != cudaSuccess) {
                rc = fail(ASDM_ERR_CUDA, "local-count gather upload failed");
                break;
            }
            const unsigned grid = (unsigned)std::min<unsigned long long>((total + 255) / 256, (unsigned long long)G->num_sms * 32);
            gather_local<<<grid, 256, 0, s>>>(d_segs, (uint32_t)segs.size(), total, d_val,
                                              reinterpret_cast<uint32_t *>(d_val + total));
            ::asdm::count_launch();
            back.resize(words);
            if (cudaGetLastError() != cudaSuccess ||
                cudaMemcpyAsync(back.data(), d_val, words * sizeof(unsigned long long), cudaMemcpyDeviceToHost, s) !=
                    cudaSuccess) {
                rc = fail(ASDM_ERR_CUDA, "local-count gather failed");
                break;
            }
        }
        fill.join();
        for (const LocalRead *r : whole)
            if (cudaMemcpyAsync(r->host, r->block, (uint64_t)G->d.n * r->cs->q.n * sizeof(unsigned long long),
                                cudaMemcpyDeviceToHost, s) != cudaSuccess)
                rc = fail(ASDM_ERR_CUDA, "local-count readback failed");
        if (cudaStreamSynchronize(s) != cudaSuccess) rc = fail(ASDM_ERR_CUDA, "local-count readback failed");
        if (rc != ASDM_OK || !total) break;
        const unsigned long long *val = back.data();
        const uint32_t *vertex = reinterpret_cast<const uint32_t *>(back.data() + total);
        constexpr uint64_t kStep = 1u << 15;
        parallel_for((total + kStep - 1) / kStep, [&](size_t k) {
            const uint64_t t0 = k * kStep, t1 = std::min<uint64_t>(total, t0 + kStep);
            size_t g = std::upper_bound(segs.begin(), segs.end(), t0,
                                        [](uint64_t t, const GatherSeg &x) { return t < x.start; }) - segs.begin() - 1;
            for (uint64_t t = t0; t < t1; ++t) {
                while (g + 1 < segs.size() && segs[g + 1].start <= t) ++g;
                host[g][(uint64_t)vertex[t] * segs[g].n + segs[g].u] = val[t];
            }
        });
    } while (false);
    dfree(d_segs, s);
    dfree(d_val, s);
    return rc;
}

}  // namespace asdm
