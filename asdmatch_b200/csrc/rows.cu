// Sorting and unpacking of embedding rows (EMBED mode).
//
// The reference prints storeMatches in sorted order (COLLECT_RESULT,
// matching/join.cpp:1032-1034).  The enumeration kernel writes every match as
// a packed key (rows.cuh); here the keys are put in order by a stable
// least-significant-digit radix sort, 8 bits a pass over the bits in use, and
// unpacked to vertex ids on the device, so that the host receives the final
// array in one copy.  A row of one word needs no permutation beside its key;
// with more words the words are sorted from the last to the first with a
// 32-bit row number each.
//
// A pass reads the keys twice (histogram, scatter) and writes them once.  At
// 6 x 10^5 six-vertex rows (7 passes) the sort's kernels take 0.2 ms and the
// copy to pageable host memory 3.7 ms; the whole call (count, enumerate, sort,
// copy) went from 203 ms with the host's sort of unpacked rows to 10 ms.
#include <algorithm>
#include <numeric>

#include "rows.cuh"

namespace asdm {
namespace {

constexpr int kSortThreads = 256, kSortWarps = kSortThreads / 32, kSortItems = 16;
constexpr int kSortTile = kSortThreads * kSortItems;
constexpr int kDigits = 256;

// Fewer rows are sorted faster on the host: the sort's 40 launches cost more
// (six columns, whole call: 2,000 rows 244 us on the host, 357 us on the
// device; 4,095 rows 408 us on the host, 4,096 rows 432 us and 5,000 rows
// 461 us on the device).
constexpr uint64_t kHostSortRows = 4096;

__global__ void __launch_bounds__(kSortThreads) digit_hist(const unsigned long long *__restrict__ key, uint64_t n,
                                                           uint32_t shift, uint64_t ntiles, uint32_t *__restrict__ hist) {
    __shared__ uint32_t h[kDigits];
    h[threadIdx.x] = 0;
    __syncthreads();
    const uint64_t base = (uint64_t)blockIdx.x * kSortTile;
#pragma unroll 4
    for (int i = 0; i < kSortItems; ++i) {
        const uint64_t r = base + (uint64_t)i * kSortThreads + threadIdx.x;
        if (r < n) atomicAdd(&h[(key[r] >> shift) & (kDigits - 1)], 1u);
    }
    __syncthreads();
    hist[(uint64_t)threadIdx.x * ntiles + blockIdx.x] = h[threadIdx.x];
}

// pos: exclusive prefix sums of hist (digit-major), so pos[d * ntiles + t] is
// where tile t's keys of digit d go.  A warp owns 512 consecutive keys of the
// tile, in 16 rounds of 32: equal digits of a round are ranked by their
// lanes, rounds by the warp's running counts, warps by a prefix over the
// warps, so the order of equal digits is kept.
template <bool kPairs>
__global__ void __launch_bounds__(kSortThreads)
    digit_scatter(const unsigned long long *__restrict__ key, const uint32_t *__restrict__ val, uint64_t n, uint32_t shift,
                  uint64_t ntiles, const uint64_t *__restrict__ pos, unsigned long long *__restrict__ key_out,
                  uint32_t *__restrict__ val_out) {
    __shared__ uint32_t cnt[kSortWarps][kDigits];
    __shared__ uint64_t first[kDigits];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (uint32_t d = lane; d < kDigits; d += 32) cnt[warp][d] = 0;
    first[threadIdx.x] = pos[(uint64_t)threadIdx.x * ntiles + blockIdx.x];
    __syncwarp();
    const uint64_t base = (uint64_t)blockIdx.x * kSortTile + warp * (32 * kSortItems) + lane;
    unsigned long long k[kSortItems];
    uint32_t rank[kSortItems];
#pragma unroll
    for (int i = 0; i < kSortItems; ++i) {
        const uint64_t r = base + 32 * i;
        k[i] = r < n ? key[r] : 0ull;
    }
#pragma unroll
    for (int i = 0; i < kSortItems; ++i) {
        const bool valid = base + 32 * i < n;
        const uint32_t active = __ballot_sync(0xffffffffu, valid);
        uint32_t before = 0, same = 0;
        const uint32_t d = (uint32_t)(k[i] >> shift) & (kDigits - 1);
        if (valid) {
            same = __match_any_sync(active, d);
            before = cnt[warp][d];
        }
        __syncwarp();
        rank[i] = before + __popc(same & ((1u << lane) - 1u));
        if (valid && (same >> lane) == 1u) cnt[warp][d] = rank[i] + 1;  // the last lane of the digit
        __syncwarp();
    }
    __syncthreads();
    {
        uint32_t run = 0;
#pragma unroll
        for (int w = 0; w < kSortWarps; ++w) {
            const uint32_t c = cnt[w][threadIdx.x];
            cnt[w][threadIdx.x] = run;
            run += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kSortItems; ++i) {
        const uint64_t r = base + 32 * i;
        if (r >= n) break;
        const uint32_t d = (uint32_t)(k[i] >> shift) & (kDigits - 1);
        const uint64_t to = first[d] + cnt[warp][d] + rank[i];
        key_out[to] = k[i];
        if (kPairs) val_out[to] = val[r];
    }
}

__global__ void iota_rows(uint32_t *__restrict__ v, uint64_t n) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        v[i] = (uint32_t)i;
}

__global__ void gather_words(const unsigned long long *__restrict__ w, const uint32_t *__restrict__ perm, uint64_t n,
                             unsigned long long *__restrict__ out) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        out[i] = w[perm[i]];
}

struct RowField {
    const uint32_t *cand;  // C(u)
    uint32_t word, shift, mask, pad;
};

// out[r * n + u] for the rows first .. first + rows - 1 (through perm, when
// given): a thread per entry, so the writes are coalesced.
__global__ void unpack_rows(const unsigned long long *__restrict__ keys, uint64_t cap, const uint32_t *__restrict__ perm,
                            uint64_t first, uint64_t rows, const RowField *__restrict__ fields, uint32_t n,
                            uint32_t *__restrict__ out) {
    const uint64_t total = rows * n;
    for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t r = t / n;
        const RowField f = fields[t - r * n];
        const uint64_t row = perm ? perm[first + r] : first + r;
        out[t] = f.cand[(uint32_t)(keys[(uint64_t)f.word * cap + row] >> f.shift) & f.mask];
    }
}

unsigned grid_of(uint64_t n, int num_sms) {
    return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((n + 255) / 256, (uint64_t)num_sms * 32));
}

struct SortBuffers {
    cudaStream_t s;
    unsigned long long *key[2] = {nullptr, nullptr};
    uint32_t *val[2] = {nullptr, nullptr};
    uint32_t *hist = nullptr;
    uint64_t *pos = nullptr;
    unsigned long long *gathered = nullptr;
    int alloc(uint64_t rows, bool pairs) {
        const uint64_t ntiles = (rows + kSortTile - 1) / kSortTile;
        for (int i = 0; i < 2; ++i) {
            ASDM_TRY(dalloc(&key[i], rows, s));
            if (pairs) ASDM_TRY(dalloc(&val[i], rows, s));
        }
        if (pairs) ASDM_TRY(dalloc(&gathered, rows, s));
        ASDM_TRY(dalloc(&hist, ntiles * kDigits, s));
        return dalloc(&pos, ntiles * kDigits + 1, s);
    }
    void release() {
        for (int i = 0; i < 2; ++i) {
            dfree(key[i], s);
            dfree(val[i], s);
        }
        dfree(hist, s);
        dfree(pos, s);
        dfree(gathered, s);
    }
    ~SortBuffers() { release(); }
};

// Sorts src (and, with values, val[*at]) by its low `bits` bits.  On return
// the keys are in *out and the values in val[*at].
int radix_sort(SortBuffers &b, const unsigned long long *src, uint64_t n, uint32_t bits, bool pairs, int *at,
               const unsigned long long **out) {
    const uint64_t ntiles = (n + kSortTile - 1) / kSortTile;
    const unsigned long long *in = src;
    int to = 0;
    for (uint32_t shift = 0; shift < bits; shift += 8) {
        digit_hist<<<(unsigned)ntiles, kSortThreads, 0, b.s>>>(in, n, shift, ntiles, b.hist);
        ::asdm::count_launch();
        ASDM_CUDA(cudaGetLastError());
        ASDM_TRY(scan_exclusive_u32(b.hist, b.pos, ntiles * kDigits, false, b.s));
        unsigned long long *ko = b.key[to];
        if (pairs) {
            digit_scatter<true><<<(unsigned)ntiles, kSortThreads, 0, b.s>>>(in, b.val[*at], n, shift, ntiles, b.pos, ko,
                                                                            b.val[*at ^ 1]);
            *at ^= 1;
        } else {
            digit_scatter<false><<<(unsigned)ntiles, kSortThreads, 0, b.s>>>(in, nullptr, n, shift, ntiles, b.pos, ko,
                                                                             nullptr);
        }
        ::asdm::count_launch();
        ASDM_CUDA(cudaGetLastError());
        in = ko;
        to ^= 1;
    }
    *out = in;
    return ASDM_OK;
}

}  // namespace

RowLayout row_layout(const asdm_cs &cs) {
    const uint32_t n = cs.q.n;
    RowLayout lay;
    lay.word.assign(n, 0);
    lay.shift.assign(n, 0);
    lay.bits.assign(n, 1);
    uint32_t used = 0;
    std::vector<uint32_t> end(n, 0);  // bits of the word in use after vertex u
    for (uint32_t u = 0; u < n; ++u) {
        while (lay.bits[u] < 32 && cs.ncand[u] > (1ull << lay.bits[u])) ++lay.bits[u];
        if (lay.words == 0 || used + lay.bits[u] > 64) {
            ++lay.words;
            lay.word_bits.push_back(0);
            used = 0;
        }
        used += lay.bits[u];
        lay.word[u] = lay.words - 1;
        lay.word_bits.back() = end[u] = used;
    }
    for (uint32_t u = 0; u < n; ++u) lay.shift[u] = lay.word_bits[lay.word[u]] - end[u];
    return lay;
}

namespace {

// The sorted rows in out, by way of the device's sort; ASDM_ERR_OOM where its
// buffers do not fit (keys are left as they were).
int device_sorted(const RowLayout &lay, const unsigned long long *keys, uint64_t cap, uint64_t rows,
                  const RowField *d_fields, uint32_t n, int num_sms, cudaStream_t s, uint32_t *out) {
    const bool pairs = lay.words > 1;
    SortBuffers b{s};
    ASDM_TRY(b.alloc(rows, pairs));
    uint32_t *d_out = nullptr;
    ASDM_TRY(dalloc(&d_out, rows * n, s));
    const unsigned long long *sorted = keys;
    uint64_t stride = cap;
    int at = 0, rc = ASDM_OK;
    if (!pairs) {
        rc = radix_sort(b, keys, rows, lay.word_bits[0], false, &at, &sorted);
        stride = rows;
    } else {
        iota_rows<<<grid_of(rows, num_sms), 256, 0, s>>>(b.val[0], rows);
        ::asdm::count_launch();
        for (uint32_t w = lay.words; w-- > 0 && rc == ASDM_OK;) {
            gather_words<<<grid_of(rows, num_sms), 256, 0, s>>>(keys + (uint64_t)w * cap, b.val[at], rows, b.gathered);
            ::asdm::count_launch();
            const unsigned long long *unused = nullptr;
            rc = radix_sort(b, b.gathered, rows, lay.word_bits[w], true, &at, &unused);
        }
    }
    if (rc == ASDM_OK) {
        unpack_rows<<<grid_of(rows * n, num_sms), 256, 0, s>>>(sorted, stride, pairs ? b.val[at] : nullptr, 0, rows,
                                                               d_fields, n, d_out);
        ::asdm::count_launch();
        if (cudaGetLastError() != cudaSuccess ||
            cudaMemcpyAsync(out, d_out, rows * n * sizeof(uint32_t), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
            cudaStreamSynchronize(s) != cudaSuccess)
            rc = fail(ASDM_ERR_CUDA, "embedding readback failed");
    }
    dfree(d_out, s);
    return rc;
}

}  // namespace

int sorted_rows(const asdm_cs &cs, const RowLayout &lay, const unsigned long long *keys, uint64_t cap, uint64_t rows,
                uint32_t *out) {
    if (rows == 0) return ASDM_OK;
    asdm_graph *G = cs.g;
    cudaStream_t s = G->stream;
    const uint32_t n = cs.q.n;
    std::vector<RowField> fields(n);
    for (uint32_t u = 0; u < n; ++u)
        fields[u] = RowField{cs.d_cand + cs.cand_base[u], lay.word[u], lay.shift[u],
                             lay.bits[u] == 32 ? 0xFFFFFFFFu : (1u << lay.bits[u]) - 1u, 0};
    RowField *d_fields = nullptr;
    uint32_t *d_out = nullptr;
    int rc = ASDM_OK;
    do {
        if ((rc = dalloc(&d_fields, n, s))) break;
        if (cudaMemcpyAsync(d_fields, fields.data(), n * sizeof(RowField), cudaMemcpyHostToDevice, s) != cudaSuccess) {
            rc = fail(ASDM_ERR_CUDA, "row layout upload failed");
            break;
        }
        // on the device where its buffers fit, row numbers fit 32 bits and tiles a grid
        if (rows >= kHostSortRows && (lay.words == 1 || rows < 0xFFFFFFFFull) && rows / kSortTile < 0x7FFFFFFFull) {
            rc = device_sorted(lay, keys, cap, rows, d_fields, n, G->num_sms, s, out);
            if (rc != ASDM_ERR_OOM) break;
        }
        // unpacked in pieces of up to 64 MiB (smaller ones where those do not
        // fit), sorted on the host
        std::vector<uint32_t> tmp(rows * n);
        uint64_t piece = std::min<uint64_t>(rows, std::max<uint64_t>(1, (16ull << 20) / n));
        while ((rc = dalloc(&d_out, piece * n, s)) == ASDM_ERR_OOM && piece > 1) piece /= 2;
        if (rc != ASDM_OK) break;
        clear_error();  // of what did not fit
        for (uint64_t r = 0; r < rows && rc == ASDM_OK; r += piece) {
            const uint64_t m = std::min(piece, rows - r);
            unpack_rows<<<grid_of(m * n, G->num_sms), 256, 0, s>>>(keys, cap, nullptr, r, m, d_fields, n, d_out);
            ::asdm::count_launch();
            if (cudaGetLastError() != cudaSuccess ||
                cudaMemcpyAsync(tmp.data() + r * n, d_out, m * n * sizeof(uint32_t), cudaMemcpyDeviceToHost, s) !=
                    cudaSuccess ||
                cudaStreamSynchronize(s) != cudaSuccess)
                rc = fail(ASDM_ERR_CUDA, "embedding readback failed");
        }
        if (rc != ASDM_OK) break;
        std::vector<uint64_t> perm(rows);
        std::iota(perm.begin(), perm.end(), 0ull);
        std::sort(perm.begin(), perm.end(), [&](uint64_t x, uint64_t y) {
            return std::lexicographical_compare(tmp.begin() + x * n, tmp.begin() + x * n + n, tmp.begin() + y * n,
                                                tmp.begin() + y * n + n);
        });
        for (uint64_t r = 0; r < rows; ++r)
            std::memcpy(out + r * n, tmp.data() + perm[r] * n, n * sizeof(uint32_t));
    } while (false);
    dfree(d_out, s);
    dfree(d_fields, s);
    cudaStreamSynchronize(s);  // the upload reads a host vector
    return rc;
}

}  // namespace asdm
