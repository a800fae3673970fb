// K1-K3: the CFL candidate space on the device.
//
// Restates CandidateSpace::buildCandCFL (relation/candidate_space.cpp:550-721)
// as the set computation it performs.  For every query vertex u, over the
// data vertices of u's label (indexed by their rank inside the label), a
// bitset F(u) holds "passes the label, degree and NLC filter" (K1, nlcValid
// at utility/utils.cpp:30-40) and one bitset per query neighbour p of u holds
// "adjacent to the storage of p" (K2).  The storage S(p) that the reference
// scans for p is the top-down candidate set Ctd(p) plus data vertex 0
// whenever Ctd(p) is smaller than |V_l(p)|: candidateSet[p] is resized to
// |V_l(p)| up front (:555-559), its zero-initialised tail is iterated by the
// range-for loops (:588, :623, :661), and pruned entries stay in it until the
// compaction at :692-703.  Hence
//     Ctd(root) = F(root),   Ctd(u) = F(u) ∩ ⋂_{p ∈ before(u)} N_l(u)(S(p)),
//     C(u) = F(u) ∩ ⋂_{p ∈ N_q(u)} N_l(u)(S(p)),
// computed wave by wave along the CFL BFS order (a vertex's wave is one more
// than the latest wave among its earlier neighbours).  The slot bitset of a
// pass p -> u is computed in pull form: a candidate's bit is set when one of
// its l(p)-neighbours lies in Ctd(p) (the phantom vertex 0 is pushed).
// Compaction ANDs the required bitsets word by word and writes the surviving
// vertices in id order.  K3 builds the candidate edges
// (buildCandidateEdge(false), :458-487) as CSR lists of indices into C(u2),
// looking a neighbour's index up in C(u2)'s membership bitset and per-word
// prefix counts.
#include <algorithm>
#include <map>
#include <memory>
#include <queue>

#include "cs.cuh"

namespace asdm {
namespace {

constexpr int kBlock = 256;
constexpr uint32_t kLongRun = 32;

__device__ __forceinline__ uint32_t find_segment(const uint64_t *__restrict__ prefix, uint32_t nseg, uint64_t item) {
    // last s with prefix[s] <= item (prefix has nseg + 1 entries, non-decreasing)
    uint32_t lo = 0, hi = nseg;
    while (hi - lo > 1) {
        uint32_t mid = (lo + hi) >> 1;
        if (prefix[mid] <= item) lo = mid; else hi = mid;
    }
    return lo;
}

// The same for a warp whose lanes hold ascending items (item = base + lane;
// lanes past the end pass valid = false, and every lane must call): the
// warp's first item is located once, 32 probes per round, and only a lane
// whose item lies past that segment searches on from there.  Segments here
// are long (a query vertex's candidates), so most warps need one search.
__device__ __forceinline__ uint32_t warp_find_segment(const uint64_t *__restrict__ prefix, uint32_t nseg,
                                                      uint64_t base, uint64_t item, bool valid, uint32_t lane) {
    uint32_t lo = 0, hi = nseg;
    while (hi - lo > 32) {
        const uint32_t step = (hi - lo + 31) / 32;
        const uint32_t p = lo + lane * step;
        const uint32_t m = __ballot_sync(0xffffffffu, p < hi && prefix[p] <= base);
        const uint32_t nlo = lo + (31 - __clz(m)) * step;
        hi = min(hi, nlo + step);
        lo = nlo;
    }
    const uint32_t p = lo + lane;
    uint32_t s = lo + (31 - __clz(__ballot_sync(0xffffffffu, p < hi && prefix[p] <= base)));
    if (valid && s + 1 < nseg && prefix[s + 1] <= item) {
        uint32_t l2 = s + 1, h2 = nseg;
        while (h2 - l2 > 1) {
            const uint32_t mid = (l2 + h2) >> 1;
            if (prefix[mid] <= item) l2 = mid; else h2 = mid;
        }
        s = l2;
    }
    return s;
}

// ---- K1: label + degree + NLC filter --------------------------------------
// One segment per (query, query vertex) of a group; a segment's items are
// the ranks 0 .. |V_l(u)| - 1 of u's label, padded to a multiple of 32 so
// that a warp's 32 items are one word of F(u).
struct FilterArgs {
    DevGraph g;
    uint32_t *bits;           // bitsets of the group
    const uint64_t *seg;      // nseg + 1 prefix of the padded item counts
    const uint64_t *fword;    // word offset of F(u) in bits
    const uint32_t *lbase;    // vbl_off[l(u)]
    const uint32_t *llen;     // |V_l(u)|
    const uint32_t *qdeg;     // deg(u)
    const uint32_t *qnlc;     // (label, count) pairs
    const uint32_t *qnlc_off; // nseg + 1
    uint32_t nq;              // number of segments
    uint32_t run_words;       // words per run
    uint32_t *fcount;         // |F(u)|
};

// A warp takes a run of up to run_words words (32 items each) inside one
// segment, so the segment lookup and the query vertex's parameters are read
// once per run: 32 words where there are enough for every warp, fewer in
// small groups (a run's words follow one another, about 1 us each: one
// 8-vertex query on 3,112 vertices took 34 us with 32).
constexpr uint32_t kMaxRunWords = 32;
// Words per warp: a power of two up to kMaxRunWords that leaves every resident warp a run.
uint32_t run_words_for(uint64_t words, int num_sms) {
    uint32_t w = kMaxRunWords;
    while (w > 1 && words < (uint64_t)num_sms * 64 * w) w >>= 1;
    return w;
}

__global__ void __launch_bounds__(kBlock) k1_filter(FilterArgs a) {
    const uint64_t total_words = a.seg[a.nq] / 32;
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t nwarps = (uint64_t)gridDim.x * (blockDim.x >> 5);
    const uint64_t nruns = (total_words + a.run_words - 1) / a.run_words;
    for (uint64_t run = (uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); run < nruns; run += nwarps) {
        uint64_t w = run * a.run_words;
        const uint64_t w_end = min(total_words, w + a.run_words);
        while (w < w_end) {
            const uint32_t u = find_segment(a.seg, a.nq, w * 32);
            const uint64_t seg_w0 = a.seg[u] / 32, seg_w1 = a.seg[u + 1] / 32;
            const uint64_t stop = min(w_end, seg_w1);
            const uint32_t len = a.llen[u], lbase = a.lbase[u], qdeg = a.qdeg[u];
            const uint32_t k0 = a.qnlc_off[u], k1 = a.qnlc_off[u + 1];
            uint32_t total = 0;
            for (; w < stop; ++w) {
                const uint32_t i = (uint32_t)(w - seg_w0) * 32 + lane;
                bool pass = false;
                if (i < len) {
                    // degree and neighbour-label mask of the vertex, in label order
                    const uint2 info = a.g.rank_info[lbase + i];
                    pass = info.x >= qdeg;
                    for (uint32_t k = k0; pass && k < k1; ++k) {
                        const uint32_t l = a.qnlc[2 * k], c = a.qnlc[2 * k + 1];
                        pass = l < a.g.nlabels && ((info.y >> (l & 31u)) & 1u);
                        if (pass && (c > 1 || a.g.nlabels > 32)) {
                            uint32_t b, e;
                            label_run(a.g, a.g.vbl[lbase + i], l, b, e);
                            pass = (e - b) >= c;
                        }
                    }
                }
                const uint32_t word = __ballot_sync(0xffffffffu, pass);
                if (lane == 0) a.bits[a.fword[u] + (w - seg_w0)] = word;
                total += __popc(word);
            }
            if (lane == 0 && total) atomicAdd(&a.fcount[u], total);
        }
    }
}

// F(u) of query vertices whose filter inputs (label, degree, neighbour-label
// counts) repeat an earlier vertex of the group: copied from that vertex's
// bitset instead of filtered again.
struct CopySeg {
    const uint32_t *src;
    uint32_t *dst;
};

__global__ void __launch_bounds__(kBlock) copy_words(const CopySeg *__restrict__ segs, const uint64_t *__restrict__ prefix,
                                                     uint32_t nseg) {
    const uint64_t total = prefix[nseg];
    for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t k = find_segment(prefix, nseg, t);
        segs[k].dst[t - prefix[k]] = segs[k].src[t - prefix[k]];
    }
}

// ---- K2: neighbour marking passes -------------------------------------------
// Pull form of a marking pass (p -> u): the bit of each candidate x of u
// (F(u) for passes from earlier BFS neighbours, Ctd(u) for the later ones:
// the final AND discards the rest) is set when some neighbour of x with label
// l(p) lies in Ctd(p).  Same bits on those candidates as pushing from S(p);
// the phantom vertex 0 of S(p), where there is one (*ph, set when Ctd(p) was
// formed: the waves run without host reads), is pushed by one more group of
// the pass, which marks its neighbours of u's label.  A warp takes a group of
// run_words words of candidates (run_words_for); each lane scans one
// candidate's label run, stopping at its first member of Ctd(p), and runs left
// open after kPullLane entries are finished by the whole warp 32 entries at a
// time.
struct PullDesc {
    const uint32_t *ph;      // whether S(p) has the phantom vertex
    const uint32_t *xbits;   // candidates to test, by rank in l(u)
    uint32_t *mbits;         // u's slot bitset for p
    const uint32_t *sbits;   // membership of Ctd(p), by rank in l(p)
    uint32_t lbase;          // vbl_off[l(u)]
    uint32_t label;          // l(p)
    uint32_t words;          // words of xbits
    uint32_t label_u;        // l(u)
};

constexpr uint32_t kPullLane = 16;

// Position of the n-th (0-based) set bit of w; n < popc(w).
__device__ __forceinline__ uint32_t nth_set_bit(uint32_t w, uint32_t n) {
    uint32_t pos = 0;
#pragma unroll
    for (uint32_t width = 16; width; width >>= 1) {
        const uint32_t low = __popc(w & ((1u << width) - 1u));
        if (n >= low) {
            n -= low;
            w >>= width;
            pos += width;
        }
    }
    return pos;
}

__device__ __forceinline__ bool pull_member(const DevGraph &g, const uint32_t *sb, uint32_t k) {
    const uint32_t z = g.nbr_rank[k];
    return (sb[z >> 5] >> (z & 31u)) & 1u;
}

__global__ void __launch_bounds__(kBlock) k2_pull(DevGraph g, const PullDesc *__restrict__ passes,
                                                  const uint64_t *__restrict__ group_pre, uint32_t npass,
                                                  uint32_t run_words, unsigned long long *__restrict__ elems) {
    constexpr uint32_t kWarps = kBlock / 32;
    __shared__ uint32_t s_out[kWarps][32];
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint64_t ngroups = group_pre[npass];
    const uint64_t nwarps = (uint64_t)gridDim.x * kWarps;
    uint64_t scanned = 0;
    s_out[wid][lane] = 0;
    __syncwarp();
    for (uint64_t grp = (uint64_t)blockIdx.x * kWarps + wid; grp < ngroups; grp += nwarps) {
        const uint32_t pi = find_segment(group_pre, npass, grp);
        const PullDesc d = passes[pi];
        const uint32_t w0 = (uint32_t)(grp - group_pre[pi]) * run_words;
        if (grp + 1 == group_pre[pi + 1]) {
            // the pass's last group: the phantom vertex
            if (*d.ph) {
                uint32_t b, e;
                label_run(g, 0, d.label_u, b, e);
                for (uint32_t k = b + lane; k < e; k += 32) {
                    const uint32_t r = g.nbr_rank[k];
                    atomicOr(&d.mbits[r >> 5], 1u << (r & 31u));  // result unused: a fire-and-forget reduction
                }
                if (lane == 0) scanned += e - b;
            }
            continue;
        }
        const uint32_t f = (lane < run_words && w0 + lane < d.words) ? d.xbits[w0 + lane] : 0u;
        // inclusive prefix of the candidates per word
        uint32_t pre = __popc(f);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, pre, o);
            if (lane >= (uint32_t)o) pre += y;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, pre, 31);
        for (uint32_t t0 = 0; t0 < total; t0 += 32) {
            const uint32_t t = t0 + lane;
            // owner word: the first lane whose inclusive prefix exceeds t
            uint32_t o = 0;
#pragma unroll
            for (uint32_t step = 16; step; step >>= 1) {
                const uint32_t v = __shfl_sync(0xffffffffu, pre, o + step - 1);
                if (v <= t) o += step;
            }
            o = min(o, 31u);
            const uint32_t word = __shfl_sync(0xffffffffu, f, o);
            const uint32_t before = __shfl_sync(0xffffffffu, pre - __popc(f), o);
            const bool mine = t < total;
            uint32_t bit = 0, b = 0, e = 0;
            if (mine) {
                bit = nth_set_bit(word, t - before);
                const uint32_t x = g.vbl[d.lbase + 32 * (w0 + o) + bit];
                label_run(g, x, d.label, b, e);
            }
            bool hit = false;
            const uint32_t stop = min(e, b + kPullLane);
            uint32_t k = b;
            for (; k < stop && !hit; ++k) hit = pull_member(g, d.sbits, k);
            scanned += k - b;
            // runs still open: the whole warp scans them
            uint32_t todo = __ballot_sync(0xffffffffu, mine && !hit && k < e);
            while (todo) {
                const int src = __ffs(todo) - 1;
                todo &= todo - 1;
                const uint32_t kk = __shfl_sync(0xffffffffu, k, src), ee = __shfl_sync(0xffffffffu, e, src);
                bool found = false;
                uint32_t seen = 0;
                for (uint32_t base = kk; base < ee && !found; base += 32) {
                    const uint32_t j = base + lane;
                    found = __any_sync(0xffffffffu, j < ee && pull_member(g, d.sbits, j));
                    seen += min(32u, ee - base);
                }
                if ((int)lane == src) {
                    hit = found;
                    scanned += seen;
                }
            }
            if (hit) atomicOr(&s_out[wid][o], 1u << bit);
        }
        __syncwarp();
        const uint32_t m = s_out[wid][lane];
        if (m) {
            atomicOr(&d.mbits[w0 + lane], m);
            s_out[wid][lane] = 0;
        }
        __syncwarp();
    }
    for (int o = 16; o; o >>= 1) scanned += __shfl_xor_sync(0xffffffffu, scanned, o);
    if (lane == 0 && scanned) atomicAdd(elems, (unsigned long long)scanned);
}

// ---- K3a: compaction of bitsets into vertex lists, word by word ------------
constexpr int kItems = 8;               // words per thread
constexpr int kTile = kBlock * kItems;  // words per tile

struct CompDesc {
    const uint32_t *bits;   // F(u); the bitset of u's query-neighbour slot b at bits + (1 + b) * words
    uint32_t words;         // ceil(|V_l(u)| / 32)
    uint32_t need;          // slots whose bitsets are required
    uint32_t len;           // |V_l(u)|
    uint32_t lbase;         // vbl_off[l(u)]
    uint2 *cmem;            // C(u): per word of the result, {membership bits, result size before it}
    uint32_t *sbits;        // Ctd(u): the result's membership bits
    uint32_t *ph;           // Ctd(u): set when fewer than len survive (the reference's zero-filled storage tail
                            // then holds data vertex 0, the phantom)
};

__device__ __forceinline__ uint32_t comp_word(const CompDesc &d, uint32_t w) {
    uint32_t x = d.bits[w];
    for (uint32_t m = d.need; m && x; m &= m - 1) x &= d.bits[(uint64_t)__ffs(m) * d.words + w];
    return x;
}

// Ctd(u) of a wave: its membership words and phantom flag.  first: prefix of
// the segments' words.
__global__ void __launch_bounds__(kBlock) k2_and(const CompDesc *__restrict__ segs, const uint64_t *__restrict__ first,
                                                 uint32_t nseg) {
    const uint64_t total = first[nseg];
    const uint32_t lane = threadIdx.x & 31;
    for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < total;
         base += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t t = base + lane;
        const uint32_t si = warp_find_segment(first, nseg, base, t, t < total, lane);
        if (t >= total) continue;
        const CompDesc d = segs[si];
        const uint32_t w = (uint32_t)(t - first[si]);
        const uint32_t x = comp_word(d, w);
        d.sbits[w] = x;
        const uint32_t left = d.len - 32 * w;  // items of this word and after it
        if (x != (left >= 32 ? 0xFFFFFFFFu : (1u << left) - 1u) && *(volatile uint32_t *)d.ph == 0) *d.ph = 1;
    }
}

__global__ void __launch_bounds__(kBlock) k3_count(const CompDesc *__restrict__ segs, const uint64_t *__restrict__ tile_first,
                                                   uint32_t nseg, uint32_t *__restrict__ tile_cnt) {
    const uint32_t t = blockIdx.x;
    const uint32_t sidx = find_segment(tile_first, nseg, t);
    const CompDesc d = segs[sidx];
    const uint32_t first = (uint32_t)(t - tile_first[sidx]) * kTile;
    uint32_t c = 0;
    for (uint32_t k = threadIdx.x; k < (uint32_t)kTile; k += kBlock) {
        const uint32_t w = first + k;
        if (w < d.words) c += __popc(comp_word(d, w));
    }
    __shared__ uint32_t wsum[kBlock / 32];
    for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0) wsum[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t s = 0;
        for (int w = 0; w < kBlock / 32; ++w) s += wsum[w];
        tile_cnt[t] = s;
    }
}

// Segment sidx writes to out + tile_pos[tile_first[sidx]].
__global__ void __launch_bounds__(kBlock) k3_write(const CompDesc *__restrict__ segs, const uint64_t *__restrict__ tile_first,
                                                   uint32_t nseg, const uint64_t *__restrict__ tile_pos,
                                                   const uint32_t *__restrict__ vbl, uint32_t *__restrict__ out,
                                                   uint32_t *__restrict__ seg_count) {
    const uint32_t t = blockIdx.x;
    const uint32_t sidx = find_segment(tile_first, nseg, t);
    const CompDesc d = segs[sidx];
    const uint32_t first = (uint32_t)(t - tile_first[sidx]) * kTile;
    const uint32_t my = first + threadIdx.x * kItems;
    uint32_t x[kItems];
    uint32_t c = 0;
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        x[k] = (my + k < d.words) ? comp_word(d, my + k) : 0u;
        c += __popc(x[k]);
    }
    // block exclusive scan of c
    __shared__ uint32_t wsum[kBlock / 32];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t v = c;
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += y;
    }
    if (lane == 31) wsum[warp] = v;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < kBlock / 32 ? wsum[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < kBlock / 32) wsum[lane] = w;
    }
    __syncthreads();
    const uint64_t seg_first = tile_pos[tile_first[sidx]];
    uint32_t *o = out + seg_first;
    uint32_t pos = (uint32_t)(tile_pos[t] - seg_first) + (warp ? wsum[warp - 1] : 0) + v - c;
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        const uint32_t w = my + k;
        if (w >= d.words) break;
        d.cmem[w] = make_uint2(x[k], pos);
        for (uint32_t y = x[k]; y; y &= y - 1) o[pos++] = vbl[d.lbase + 32 * w + (uint32_t)(__ffs(y) - 1)];
    }
    // the last tile of a segment records the segment size
    if (threadIdx.x == 0 && t + 1 == tile_first[sidx + 1]) seg_count[sidx] = (uint32_t)(tile_pos[t + 1] - seg_first);
}

// ---- K3b: candidate edges ---------------------------------------------------
struct EdgeDesc {
    const uint32_t *cand_u;   // C(u)
    uint32_t cmem;            // offset in the group's membership words: per word of ranks in l(u2),
                              // {membership of C(u2), |C(u2)| before it}
    uint32_t ncand_u;
    uint32_t label_u2;
    uint32_t pad;
};

// Index in C(u2) of the vertex of rank r in l(u2), or kNone (one 8-byte
// load: the word's bits and prefix side by side).
__device__ __forceinline__ uint32_t cand_index(const uint2 *cm, uint32_t r) {
    const uint2 w = cm[r >> 5];
    const uint32_t bit = 1u << (r & 31u);
    return (w.x & bit) ? w.y + (uint32_t)__popc(w.x & (bit - 1u)) : kNone;
}

// Every item's list in one scan of its label run: its length in cnt, or (kFill)
// its entries at elist + wpos[item].
template <bool kFill>
__global__ void __launch_bounds__(kBlock) k3_edges(DevGraph g, const EdgeDesc *__restrict__ edges,
                                                   const uint2 *__restrict__ cmem,
                                                   const uint64_t *__restrict__ item_base, uint32_t nedges,
                                                   uint32_t *__restrict__ cnt, const uint64_t *__restrict__ wpos,
                                                   uint32_t *__restrict__ elist,
                                                   unsigned long long *__restrict__ elems) {
    const uint64_t total = item_base[nedges];
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    uint64_t scanned = 0;
    for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < total; base += stride) {
        const uint64_t pos = base + lane;
        const uint64_t item = pos;
        uint32_t b = 0, e = 0;
        const uint2 *cm = nullptr;
        const uint32_t ei = warp_find_segment(item_base, nedges, base, item, pos < total, lane);
        if (pos < total) {
            const EdgeDesc d = edges[ei];
            const uint32_t i = (uint32_t)(item - item_base[ei]);
            if (i < d.ncand_u) label_run(g, d.cand_u[i], d.label_u2, b, e);
            cm = cmem + d.cmem;
        }
        scanned += e - b;
        const bool coop = (e - b) > kLongRun;
        uint32_t mine = 0;
        uint64_t out = kFill && pos < total ? wpos[item] : 0;
        uint32_t todo = __ballot_sync(0xffffffffu, coop);
        while (todo) {
            const int src = __ffs(todo) - 1;
            todo &= todo - 1;
            const uint32_t bb = __shfl_sync(0xffffffffu, b, src), ee = __shfl_sync(0xffffffffu, e, src);
            const uint2 *mm = (const uint2 *)__shfl_sync(0xffffffffu, (unsigned long long)cm, src);
            uint64_t o = __shfl_sync(0xffffffffu, out, src);
            uint32_t c = 0;
            for (uint32_t k0 = bb; k0 < ee; k0 += 32) {
                const uint32_t k = k0 + lane;
                const uint32_t idx = k < ee ? cand_index(mm, g.nbr_rank[k]) : kNone;
                const uint32_t hit = __ballot_sync(0xffffffffu, idx != kNone);
                if (kFill && idx != kNone) elist[o + __popc(hit & ((1u << lane) - 1))] = idx;
                o += __popc(hit);
                c += __popc(hit);
            }
            if ((int)lane == src) mine = c;
        }
        if (!coop) {
#pragma unroll 4
            for (uint32_t k = b; k < e; ++k) {
                const uint32_t idx = cand_index(cm, g.nbr_rank[k]);
                if (idx != kNone) {
                    if (kFill) elist[out++] = idx;
                    ++mine;
                }
            }
        }
        if (cnt && pos < total) cnt[item] = mine;
    }
    if (elems) {
        for (int o = 16; o; o >>= 1) scanned += __shfl_xor_sync(0xffffffffu, scanned, o);
        if (lane == 0 && scanned) atomicAdd(elems, (unsigned long long)scanned);
    }
}

// The fill: every item's label run is scanned once.
//
// The entries of all runs, in item order, are cut into chunks of equal length, a
// warp each, so hubs' runs spread over many warps.  A warp walks its chunk 32
// entries at a time, a lane per entry, kRounds rounds' loads in flight
// together; the items that start in a round are one bit mask (a warp
// reduction), so an entry's owner is a population count.  Entries are in
// output order, so the hits, packed by ballots, are the chunk's part of the
// output as it stands: they go to the chunk's own place in a staging buffer,
// and a prefix sum over the chunks' hits says where k3_pack copies them.
//
// Bound: the two dependent loads per entry (neighbour rank, membership word;
// L2 hits mostly) and the instructions around them.  Measured on 512 queries
// on 3.77M vertices (1.2 x 10^10 entries, 8.4 x 10^9 hits): a binary search
// for every entry's owner in 64-bit positions 135 ms (and 36 ms for a packing
// pass per item); tiles of a fixed number of items 275 ms (every block waits
// for its hubs); chunks written at their final place after a look-back over
// the chunks before them 84 ms with a look-back per block, 98 ms per warp
// (thousands of chunks in flight to walk over).
constexpr uint32_t kRounds = 4;
// Entries per chunk, a power of two: finding its first items costs a chunk a
// few dependent loads (512 queries as above: 83 ms with 512 entries, 69 ms
// with 1,024, 61 ms with 2,048), but a small group needs its warps spread
// (200 8-vertex queries on 3,112 vertices, 51,000 entries: 24 us with 512
// entries, 63 us with 2,048), so chunks grow once every warp has two.
constexpr uint32_t kChunkLog2Min = 7, kChunkLog2Max = 12;
uint32_t chunk_log2_for(uint64_t entries, int num_sms) {
    uint32_t k = kChunkLog2Min;
    while (k < kChunkLog2Max && entries >> (k + 1) >= (uint64_t)num_sms * 64 * 2) ++k;
    return k;
}

struct FillWarp {
    uint2 item[32];  // by rank among the batch's non-empty items: {entry number -> place in nbr_rank, cmem offset}
};

// The hits of 32 items (lane's item: entries nbr_rank[rs, rs + len),
// membership words at cmem + cm), packed behind out; off = hits before this
// lane's item.  Returns their number.
__device__ __forceinline__ uint32_t fill_batch(const uint32_t *__restrict__ nbr_rank, const uint2 *__restrict__ cmem,
                                               FillWarp &w, uint32_t lane, uint32_t rs, uint32_t len, uint32_t cm,
                                               uint32_t *__restrict__ out, uint32_t &off) {
    uint32_t inc = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= (uint32_t)o) inc += y;
    }
    const uint32_t start = inc - len, S = __shfl_sync(0xffffffffu, inc, 31);
    const uint32_t lt = (1u << lane) - 1u, le = lt | (1u << lane);
    const uint32_t some = __ballot_sync(0xffffffffu, len != 0);
    if (len) w.item[__popc(some & lt)] = make_uint2(rs - start, cm);
    __syncwarp();
    uint32_t hits = 0, seen = 0;  // hits so far, non-empty items started so far
    for (uint32_t j0 = 0; j0 < S; j0 += 32 * kRounds) {
        uint2 it[kRounds], wd[kRounds];
        uint32_t rank[kRounds];
#pragma unroll
        for (uint32_t r = 0; r < kRounds; ++r) {
            const uint32_t d = start - (j0 + 32 * r);  // 32 or more when not in the round
            const uint32_t heads = __reduce_or_sync(0xffffffffu, len && d < 32 ? 1u << d : 0u);
            it[r] = w.item[seen + __popc(heads & le) - 1];
            seen += __popc(heads);
        }
#pragma unroll
        for (uint32_t r = 0; r < kRounds; ++r)  // lanes past the end repeat the last entry
            rank[r] = nbr_rank[min(j0 + 32 * r + lane, S - 1) + it[r].x];
#pragma unroll
        for (uint32_t r = 0; r < kRounds; ++r) wd[r] = cmem[it[r].y + (rank[r] >> 5)];
#pragma unroll
        for (uint32_t r = 0; r < kRounds; ++r) {
            const uint32_t bit = rank[r] & 31u;
            const bool hit = ((wd[r].x >> bit) & 1u) && j0 + 32 * r + lane < S;
            const uint32_t m = __ballot_sync(0xffffffffu, hit);
            const uint32_t d = start - (j0 + 32 * r);
            if (d < 32) off = hits + __popc(m & ((1u << d) - 1u));
            if (hit) out[hits + __popc(m & lt)] = wd[r].y + __popc(wd[r].x & ((1u << bit) - 1u));
            hits += __popc(m);
        }
    }
    if (start >= S) off = hits;  // empty items after the last entry
    __syncwarp();
    return hits;
}

// The first item of every chunk (the one whose run holds the chunk's first
// entry, or the first of the empty items at that place) and its edge.
__global__ void __launch_bounds__(kBlock) k3_chunks(const uint64_t *__restrict__ item_base, uint32_t nedges,
                                                    const uint64_t *__restrict__ upos, uint32_t chunk_log2,
                                                    uint2 *__restrict__ chunk) {
    const uint64_t total = item_base[nedges];
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t s = upos[i], e = upos[i + 1];
        uint64_t c = (s + (1ull << chunk_log2) - 1) >> chunk_log2;
        if (c << chunk_log2 >= e) continue;
        uint32_t f = (uint32_t)i, ei = find_segment(item_base, nedges, i);
        for (; c << chunk_log2 < e; ++c) {
            if (c << chunk_log2 == s) {
                uint32_t b = f;
                while (b > 0 && upos[b - 1] == s) --b;
                chunk[c] = make_uint2(b, b == f ? ei : find_segment(item_base, nedges, b));
            } else {
                chunk[c] = make_uint2(f, ei);
            }
        }
    }
}

// In: upos = prefix of the run lengths (nitems + 1), rstart = run starts, the
// chunks' first items.  Out: the chunks' hits in stage, their numbers; eoff =
// each item's position among its chunk's hits.
__global__ void __launch_bounds__(kBlock, 5) k3_fill(DevGraph g, const EdgeDesc *__restrict__ edges,
                                                  const uint2 *__restrict__ cmem,
                                                  const uint64_t *__restrict__ item_base, uint32_t nedges,
                                                  const uint64_t *__restrict__ upos, const uint32_t *__restrict__ rstart,
                                                  const uint2 *__restrict__ chunk, uint32_t nchunks, uint32_t chunk_log2,
                                                  uint32_t *__restrict__ eoff, uint32_t *__restrict__ stage,
                                                  uint32_t *__restrict__ chunk_hits) {
    __shared__ FillWarp s_warp[kBlock / 32];
    const uint32_t lane = threadIdx.x & 31;
    FillWarp &w = s_warp[threadIdx.x >> 5];
    const uint32_t nitems = (uint32_t)item_base[nedges];
    const uint64_t entries = upos[nitems];
    const uint64_t nwarps = (uint64_t)gridDim.x * (kBlock / 32);
    for (uint64_t c = (uint64_t)blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5); c < nchunks; c += nwarps) {
        const bool last = c + 1 == nchunks;
        const uint64_t e0 = c << chunk_log2, e1 = last ? entries : e0 + (1ull << chunk_log2);
        const uint2 p = chunk[c];
        uint32_t base = p.x, edge = p.y, hits = 0;
        uint64_t edge_end = item_base[edge + 1];
        uint64_t s = base + lane < nitems ? upos[base + lane] : entries;
        uint32_t rs = base + lane < nitems ? rstart[base + lane] : 0u;
        for (;;) {
            const uint32_t item = base + lane;
            // the next 32 items, in flight while these are scanned
            const bool more = (uint64_t)item + 32 < nitems;
            const uint64_t s_next = more ? upos[item + 32] : entries;
            const uint32_t rs_next = more ? rstart[item + 32] : 0u;
            // this lane's edge: the warp's, or one of the next
            uint32_t ei = edge;
            if (item >= edge_end && item < nitems) ei = find_segment(item_base + edge, min(32u, nedges - edge), item) + edge;
            const uint32_t cm = edges[ei].cmem;
            const uint64_t after = __shfl_sync(0xffffffffu, s_next, 0);
            uint64_t e = __shfl_down_sync(0xffffffffu, s, 1);
            if (lane == 31) e = after;
            const uint64_t lo = max(s, e0), hi = min(e, e1);
            const uint32_t len = hi > lo ? (uint32_t)(hi - lo) : 0u;
            uint32_t off = 0;
            const uint32_t h = fill_batch(g.nbr_rank, cmem, w, lane, rs + (uint32_t)(lo - s), len, cm, stage + e0 + hits, off);
            if (item < nitems && s >= e0 && (s < e1 || last)) eoff[item] = hits + off;
            hits += h;
            if ((uint64_t)base + 32 >= nitems || (after >= e1 && !last)) break;
            base += 32;
            s = s_next;
            rs = rs_next;
            edge = __shfl_sync(0xffffffffu, ei, 31);
            edge_end = item_base[edge + 1];
            if (edge_end <= base) edge_end = item_base[++edge + 1];  // lane 31 was its edge's last item
        }
        if (lane == 0) chunk_hits[c] = hits;
    }
}

// The chunks' hits, side by side in elist: a warp per chunk, four entries a
// lane in flight.
__global__ void __launch_bounds__(kBlock) k3_pack(const uint32_t *__restrict__ stage, const uint32_t *__restrict__ chunk_hits,
                                                  const uint64_t *__restrict__ chunk_base, uint32_t nchunks,
                                                  uint32_t chunk_log2, uint32_t *__restrict__ elist) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t nwarps = (uint64_t)gridDim.x * (kBlock / 32);
    for (uint64_t c = (uint64_t)blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5); c < nchunks; c += nwarps) {
        const uint32_t n = chunk_hits[c];
        const uint32_t *from = stage + (c << chunk_log2);
        uint32_t *to = elist + chunk_base[c];
        for (uint32_t i = lane; i < n; i += 128) {
            uint32_t v[4];
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k) v[k] = i + 32 * k < n ? from[i + 32 * k] : 0u;
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k)
                if (i + 32 * k < n) to[i + 32 * k] = v[k];
        }
    }
}

// Where an item's list starts in elist, from k3_fill's outputs.
__device__ __forceinline__ unsigned long long list_start(const uint64_t *upos, uint32_t nchunks, uint32_t chunk_log2,
                                                         const uint64_t *chunk_base, const uint32_t *eoff,
                                                         uint64_t item) {
    const uint64_t c = upos[item] >> chunk_log2;
    return chunk_base[c < nchunks ? c : nchunks - 1] + eoff[item];
}

__global__ void k3_starts(const uint64_t *__restrict__ item_base, uint32_t nedges, const uint64_t *__restrict__ upos,
                          uint32_t nchunks, uint32_t chunk_log2, const uint64_t *__restrict__ chunk_base,
                          const uint32_t *__restrict__ eoff, uint64_t *__restrict__ edge_start) {
    const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e < nedges) edge_start[e] = list_start(upos, nchunks, chunk_log2, chunk_base, eoff, item_base[e]);
}

// eoff relative to its edge's first entry (below 2^32: checked by the host)
__global__ void __launch_bounds__(kBlock) k3_rebase(const uint64_t *__restrict__ item_base, uint32_t nedges,
                                                    const uint64_t *__restrict__ upos, uint32_t nchunks, uint32_t chunk_log2,
                                                    const uint64_t *__restrict__ chunk_base,
                                                    const uint64_t *__restrict__ edge_start, uint32_t *__restrict__ eoff) {
    const uint64_t total = item_base[nedges];
    const uint32_t lane = threadIdx.x & 31;
    for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < total;
         base += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t i = base + lane;
        const uint32_t ei = warp_find_segment(item_base, nedges, base, i, i < total, lane);
        if (i < total) eoff[i] = (uint32_t)(list_start(upos, nchunks, chunk_log2, chunk_base, eoff, i) - edge_start[ei]);
    }
}

// Every item's label run: its length (the upper bound of its list) and start.
__global__ void __launch_bounds__(kBlock) k3_bound(DevGraph g, const EdgeDesc *__restrict__ edges,
                                                   const uint64_t *__restrict__ item_base, uint32_t nedges,
                                                   uint32_t *__restrict__ ub, uint32_t *__restrict__ rstart) {
    const uint64_t total = item_base[nedges];
    const uint32_t lane = threadIdx.x & 31;
    for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < total;
         base += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t item = base + lane;
        const uint32_t ei = warp_find_segment(item_base, nedges, base, item, item < total, lane);
        if (item >= total) continue;
        const EdgeDesc d = edges[ei];
        const uint32_t i = (uint32_t)(item - item_base[ei]);
        uint32_t b = 0, e = 0;
        if (i < d.ncand_u) label_run(g, d.cand_u[i], d.label_u2, b, e);
        ub[item] = e - b;
        rstart[item] = b;
    }
}

__global__ void k3_offsets(const uint64_t *__restrict__ item_base, uint32_t nedges, const uint64_t *__restrict__ wpos,
                           uint32_t *__restrict__ eoff, uint64_t *__restrict__ edge_start, uint32_t *__restrict__ bad) {
    const uint64_t total = item_base[nedges];
    const uint32_t lane = threadIdx.x & 31;
    for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < total;
         base += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t i = base + lane;
        const uint32_t ei = warp_find_segment(item_base, nedges, base, i, i < total, lane);
        if (i >= total) continue;
        const uint64_t rel = wpos[i] - wpos[item_base[ei]];
        if (rel > 0xFFFFFFFFull) atomicExch(bad, 1u);
        eoff[i] = (uint32_t)rel;
        if (i == item_base[ei]) edge_start[ei] = wpos[i];
    }
}

unsigned grid_for(uint64_t items, int num_sms) {
    uint64_t blocks = (items + kBlock - 1) / kBlock;
    return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(blocks, (uint64_t)num_sms * 32));
}

// Candidate arrays of at most this many entries in total are allocated for
// their bound, |V_l(u)| each, so the host need not read their sizes first.
constexpr uint64_t kCandBound = 1u << 20;
// Items and possible list entries of a group small enough for K3's short form,
// and the possible entries whose memory (4 MiB) is not worth a readback.
constexpr uint64_t kSmallItems = 1u << 16, kSmallLists = 1u << 22, kListBound = 1u << 20;

struct Scratch {
    cudaStream_t s;
    asdm_graph *G;
    std::vector<void *> ptrs;
    ~Scratch() {
        for (void *p : ptrs) cudaFreeAsync(p, s);
    }
    template <typename T>
    int alloc(T **p, uint64_t n) {
        int rc = dalloc(p, n, s);
        if (rc == ASDM_OK) ptrs.push_back((void *)*p);
        return rc;
    }
};

// Descriptor arrays that go to the device in one allocation and one copy
// (a copy costs the host about 5 us whatever its size).
struct Blob {
    std::vector<uint8_t> h;
    uint8_t *d = nullptr;
    template <typename T>
    size_t put(const std::vector<T> &v) {
        const size_t at = (h.size() + 15) & ~size_t(15);
        h.resize(at + v.size() * sizeof(T));
        if (!v.empty()) std::memcpy(h.data() + at, v.data(), v.size() * sizeof(T));
        return at;
    }
    size_t zeros(size_t bytes) {
        const size_t at = (h.size() + 15) & ~size_t(15);
        h.resize(at + bytes, 0);
        return at;
    }
    int upload(Scratch &scr) {
        ASDM_TRY(scr.alloc(&d, h.size()));
        if (!h.empty()) ASDM_CUDA(upload_async(scr.G, d, h.data(), h.size()));
        return ASDM_OK;
    }
    template <typename T>
    T *at(size_t o) const {
        return reinterpret_cast<T *>(d + o);
    }
};

// Host-side plan of one query's CFL build.
struct QPlan {
    asdm_cs *cs;
    uint32_t seg0;                  // first segment (query vertex 0)
    bool empty = false;
    std::vector<uint32_t> lsize, lbase, rank, order, wave;
};

}  // namespace

// Candidate spaces of a group of queries on one graph, one launch per phase
// for the whole group.  Every phase is the single-query computation applied
// to all (query, query vertex) segments at once.
int build_batch(const std::vector<asdm_cs *> &group) {
    if (group.empty()) return ASDM_OK;
    asdm_graph *G = group[0]->g;
    const DevGraph &g = G->d;
    cudaStream_t s = G->stream;
    Scratch scr{s, G, {}};
    // descriptor uploads go through the graph's pinned stage, reused per build
    ASDM_CUDA(cudaStreamSynchronize(s));
    G->stage.reset();
    cudaEvent_t ev0, ev1;
    ASDM_CUDA(cudaEventCreate(&ev0));
    ASDM_CUDA(cudaEventCreate(&ev1));
    ASDM_CUDA(cudaEventRecord(ev0, s));
    const uint32_t Q = (uint32_t)group.size();
    std::vector<QPlan> P(Q);
    uint32_t nseg = 0;
    for (uint32_t qi = 0; qi < Q; ++qi) {
        QPlan &qp = P[qi];
        qp.cs = group[qi];
        const QueryGraph &q = qp.cs->q;
        qp.seg0 = nseg;
        nseg += q.n;
        qp.lsize.assign(q.n, 0);
        qp.lbase.assign(q.n, 0);
        for (uint32_t u = 0; u < q.n; ++u) {
            const uint32_t l = q.lab[u];
            if (l < g.nlabels) {
                qp.lbase[u] = G->h_vbl_off[l];
                qp.lsize[u] = G->h_vbl_off[l + 1] - G->h_vbl_off[l];
            }
        }
    }
    // bitset layout [F | slot 0 | slot 1 | ...] per query vertex; K1 filters
    // one query vertex per distinct (label, degree, neighbour-label counts)
    // and copies F to the others
    std::vector<uint64_t> fword(nseg + 1, 0);
    std::vector<uint32_t> words(nseg);
    std::vector<uint64_t> seg{0}, kfword;               // K1 segments (distinct signatures)
    std::vector<uint32_t> lbase, llen, qdeg, qnlc, qnlc_off{0};
    std::map<std::vector<uint32_t>, uint32_t> sig_k1;   // signature -> K1 segment
    std::vector<uint32_t> k1_of(nseg);
    for (const QPlan &qp : P) {
        const QueryGraph &q = qp.cs->q;
        for (uint32_t u = 0; u < q.n; ++u) {
            const uint32_t sg = qp.seg0 + u;
            words[sg] = (qp.lsize[u] + 31) / 32;
            fword[sg + 1] = fword[sg] + (uint64_t)(q.deg(u) + 1) * words[sg];
            std::vector<uint32_t> sig{q.lab[u], q.deg(u)};
            for (uint32_t e = q.off[u]; e < q.off[u + 1]; ++e) {
                const uint32_t l = q.lab[q.nbr[e]];
                if (sig.size() > 2 && sig[sig.size() - 2] == l) sig.back()++;
                else { sig.push_back(l); sig.push_back(1); }
            }
            auto it = sig_k1.find(sig);
            if (it != sig_k1.end()) {
                k1_of[sg] = it->second;
                continue;
            }
            const uint32_t k = (uint32_t)lbase.size();
            sig_k1.emplace(sig, k);
            k1_of[sg] = k;
            seg.push_back(seg.back() + 32ull * words[sg]);
            kfword.push_back(fword[sg]);
            lbase.push_back(qp.lbase[u]);
            llen.push_back(qp.lsize[u]);
            qdeg.push_back(q.deg(u));
            qnlc.insert(qnlc.end(), sig.begin() + 2, sig.end());
            qnlc_off.push_back((uint32_t)(qnlc.size() / 2));
        }
    }
    const uint32_t nk1 = (uint32_t)lbase.size();
    kfword.push_back(0);
    uint32_t *bits = nullptr;
    ASDM_TRY(scr.alloc(&bits, fword[nseg]));
    ASDM_CUDA(cudaMemsetAsync(bits, 0, std::max<uint64_t>(fword[nseg], 1) * sizeof(uint32_t), s));
    // F of the repeated signatures
    std::vector<CopySeg> cps;
    std::vector<uint64_t> cpre{0};
    for (uint32_t sg = 0; sg < nseg; ++sg) {
        const uint32_t k = k1_of[sg];
        if (kfword[k] == fword[sg]) continue;  // the vertex K1 filtered
        cps.push_back(CopySeg{bits + kfword[k], bits + fword[sg]});
        cpre.push_back(cpre.back() + words[sg]);
    }
    const uint64_t copied_words = cpre.back();
    Blob b1;
    const size_t o_seg = b1.put(seg), o_fword = b1.put(kfword), o_lbase = b1.put(lbase), o_llen = b1.put(llen),
                 o_qdeg = b1.put(qdeg), o_qnlc = b1.put(qnlc), o_qnlc_off = b1.put(qnlc_off), o_cps = b1.put(cps),
                 o_cpre = b1.put(cpre), o_fcount = b1.zeros(std::max<uint32_t>(nk1, 1) * sizeof(uint32_t)),
                 o_elems = b1.zeros(2 * sizeof(unsigned long long)),
                 o_ph = b1.zeros(std::max<uint32_t>(nseg, 1) * sizeof(uint32_t)), o_bad = b1.zeros(sizeof(uint32_t));
    ASDM_TRY(b1.upload(scr));
    uint32_t *d_fcount = b1.at<uint32_t>(o_fcount), *d_ph = b1.at<uint32_t>(o_ph);
    unsigned long long *d_elems = b1.at<unsigned long long>(o_elems);
    if (seg[nk1]) {
        const uint64_t kwords = seg[nk1] / 32;
        const uint32_t rw = run_words_for(kwords, G->num_sms);
        FilterArgs fa{g, bits, b1.at<uint64_t>(o_seg), b1.at<uint64_t>(o_fword), b1.at<uint32_t>(o_lbase),
                      b1.at<uint32_t>(o_llen), b1.at<uint32_t>(o_qdeg), b1.at<uint32_t>(o_qnlc),
                      b1.at<uint32_t>(o_qnlc_off), nk1, rw, d_fcount};
        k1_filter<<<grid_for((kwords + rw - 1) / rw * 32, G->num_sms), kBlock, 0, s>>>(fa);  // a warp per run
        ::asdm::count_launch();
        ASDM_CUDA(cudaGetLastError());
    }
    if (copied_words) {
        copy_words<<<grid_for(copied_words, G->num_sms), kBlock, 0, s>>>(b1.at<CopySeg>(o_cps), b1.at<uint64_t>(o_cpre),
                                                                        (uint32_t)cps.size());
        ::asdm::count_launch();
        ASDM_CUDA(cudaGetLastError());
    }
    std::vector<uint32_t> kcount(std::max<uint32_t>(nk1, 1), 0), fcount(nseg, 0);
    ASDM_CUDA(cudaMemcpyAsync(kcount.data(), d_fcount, kcount.size() * sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    ASDM_CUDA(cudaStreamSynchronize(s));
    for (uint32_t sg = 0; sg < nseg; ++sg) fcount[sg] = kcount[k1_of[sg]];

    uint32_t maxwave = 0;
    for (QPlan &qp : P) {
        asdm_cs &cs = *qp.cs;
        const QueryGraph &q = cs.q;
        const uint32_t nq = q.n;
        // Root: the three smallest |V_l(u)|/deg(u) kept in a max-heap, then the
        // first strict minimum of |F(u)|/deg(u) in pop order (selectCFLRoot,
        // relation/candidate_space.cpp:723-763; same container and comparator).
        auto cmp = [](const std::pair<uint32_t, double> &x, const std::pair<uint32_t, double> &y) {
            return x.second < y.second;
        };
        std::priority_queue<std::pair<uint32_t, double>, std::vector<std::pair<uint32_t, double>>, decltype(cmp)> pq(cmp);
        for (uint32_t u = 0; u < nq; ++u) pq.emplace(u, qp.lsize[u] / (double)q.deg(u));
        while (pq.size() > 3) pq.pop();
        uint32_t root = 0;
        double best = g.n;
        while (!pq.empty()) {
            const uint32_t u = pq.top().first;
            pq.pop();
            const double score = fcount[qp.seg0 + u] / (double)q.deg(u);
            if (score < best) { best = score; root = u; }
        }
        cs.root = root;
        // BFS levels with discovery order over (label,id)-sorted query
        // neighbours (buildCFLBFSTree, :765-816); rank = position in that order
        qp.rank.assign(nq, kNone);
        qp.order.clear();
        std::vector<uint32_t> frontier{root};
        qp.rank[root] = 0;
        uint32_t r = 1;
        while (!frontier.empty()) {
            std::vector<uint32_t> next;
            for (uint32_t u : frontier) {
                qp.order.push_back(u);
                for (uint32_t e = q.off[u]; e < q.off[u + 1]; ++e) {
                    const uint32_t w = q.nbr[e];
                    if (qp.rank[w] == kNone) { qp.rank[w] = r++; next.push_back(w); }
                }
            }
            frontier.swap(next);
        }
        cs.bfs_order = qp.order;
        cs.ncand.assign(nq, 0);
        cs.cand_base.assign(nq + 1, 0);
        cs.nonempty = false;
        qp.empty = qp.order.size() != nq;  // unreached query vertices get no candidates
        for (uint32_t u = 0; u < nq; ++u) qp.empty |= fcount[qp.seg0 + u] == 0;
        qp.wave.assign(nq, 0);
        if (qp.empty) continue;
        for (uint32_t u : qp.order) {
            for (uint32_t e = q.off[u]; e < q.off[u + 1]; ++e) {
                const uint32_t p = q.nbr[e];
                if (qp.rank[p] < qp.rank[u]) qp.wave[u] = std::max(qp.wave[u], qp.wave[p] + 1);
            }
            maxwave = std::max(maxwave, qp.wave[u]);
        }
    }
    // Ctd(u) as a membership bitset per query vertex (and whether the
    // storage S(u) scanned by the reference gets the phantom vertex 0)
    std::vector<uint64_t> mword(nseg + 1, 0);
    for (uint32_t i = 0; i < nseg; ++i) mword[i + 1] = mword[i] + words[i];
    // (d_ph).  The waves' descriptors, the later passes' and the final
    // compaction's go up together: no host read lies between them.
    uint32_t *sbits = nullptr;
    uint2 *cmem = nullptr;
    ASDM_TRY(scr.alloc(&sbits, std::max<uint64_t>(mword[nseg], 1)));
    ASDM_TRY(scr.alloc(&cmem, mword[nseg]));
    uint64_t bit_words_read = 0;
    struct Wave {
        uint32_t npull = 0, nand = 0, run_words = 1;
        uint64_t groups = 0, words = 0;
        size_t o_pull = 0, o_gpre = 0, o_and = 0, o_wpre = 0;
    };
    Blob b2;
    std::vector<PullDesc> pulls;
    // a pass p -> u, pulled over u's candidates (and the phantom's push)
    auto add_pass = [&](const QPlan &qp, uint32_t u, uint32_t e, const uint32_t *xbits) {
        const QueryGraph &q = qp.cs->q;
        const uint32_t p = q.nbr[e], su = qp.seg0 + u, sp = qp.seg0 + p, slot = e - q.off[u];
        uint32_t *mb = bits + fword[su] + (1ull + slot) * words[su];
        pulls.push_back(PullDesc{d_ph + sp, xbits, mb, sbits + mword[sp], qp.lbase[u], q.lab[p], words[su], q.lab[u]});
        bit_words_read += words[su];
    };
    auto put_pulls = [&](Wave &wv) {
        uint64_t all = 0;
        for (const PullDesc &d : pulls) all += d.words;
        wv.run_words = run_words_for(all, G->num_sms);
        std::vector<uint64_t> gpre{0};
        for (const PullDesc &d : pulls) gpre.push_back(gpre.back() + (d.words + wv.run_words - 1) / wv.run_words + 1);
        wv.npull = (uint32_t)pulls.size();
        wv.groups = gpre.back();
        wv.o_pull = b2.put(pulls);
        wv.o_gpre = b2.put(gpre);
        pulls.clear();
    };
    std::vector<Wave> waves(maxwave + 2);
    for (uint32_t w = 0; w <= maxwave; ++w) {
        std::vector<CompDesc> ands;
        std::vector<uint64_t> wpre{0};
        for (const QPlan &qp : P) {
            if (qp.empty) continue;
            const QueryGraph &q = qp.cs->q;
            for (uint32_t u : qp.order) {
                if (qp.wave[u] != w) continue;
                const uint32_t su = qp.seg0 + u;
                uint32_t need = 0;
                for (uint32_t e = q.off[u]; e < q.off[u + 1]; ++e) {
                    if (qp.rank[q.nbr[e]] >= qp.rank[u]) continue;
                    need |= 1u << (e - q.off[u]);
                    add_pass(qp, u, e, bits + fword[su]);  // over F(u)
                }
                ands.push_back(CompDesc{bits + fword[su], words[su], need, qp.lsize[u], qp.lbase[u], nullptr,
                                        sbits + mword[su], d_ph + su});
                wpre.push_back(wpre.back() + words[su]);
                bit_words_read += (uint64_t)(1 + __builtin_popcount(need)) * words[su];
            }
        }
        put_pulls(waves[w]);
        waves[w].nand = (uint32_t)ands.size();
        waves[w].words = wpre.back();
        waves[w].o_and = b2.put(ands);
        waves[w].o_wpre = b2.put(wpre);
    }
    // remaining passes (neighbours later in the BFS order), all queries at
    // once, over Ctd(u); then the final candidate sets, with the membership
    // words and per-word prefix counts that K3 looks indices up in
    std::vector<CompDesc> segs;
    std::vector<uint32_t> seg_ids;
    std::vector<uint64_t> tile_first{0};
    uint64_t cand_bound = 0;
    for (const QPlan &qp : P) {
        if (qp.empty) continue;
        const QueryGraph &q = qp.cs->q;
        for (uint32_t u = 0; u < q.n; ++u) {
            const uint32_t su = qp.seg0 + u;
            for (uint32_t e = q.off[u]; e < q.off[u + 1]; ++e)
                if (qp.rank[q.nbr[e]] >= qp.rank[u]) add_pass(qp, u, e, sbits + mword[su]);
            const uint32_t all = q.deg(u) ? ((q.deg(u) == 32 ? 0xFFFFFFFFu : (1u << q.deg(u)) - 1u)) : 0u;
            segs.push_back(CompDesc{bits + fword[su], words[su], all, qp.lsize[u], qp.lbase[u], cmem + mword[su],
                                    nullptr, nullptr});
            seg_ids.push_back(su);
            tile_first.push_back(tile_first.back() + (words[su] + kTile - 1) / kTile);
            cand_bound += qp.lsize[u];
            bit_words_read += (uint64_t)(1 + q.deg(u)) * words[su];
        }
    }
    put_pulls(waves[maxwave + 1]);
    const uint32_t nfinal = (uint32_t)segs.size();
    const uint64_t ntiles = tile_first.back();
    const size_t o_segs = b2.put(segs), o_tf = b2.put(tile_first);
    ASDM_TRY(b2.upload(scr));
    for (const Wave &wv : waves) {
        if (wv.npull) {
            k2_pull<<<grid_for(32 * wv.groups, G->num_sms), kBlock, 0, s>>>(g, b2.at<PullDesc>(wv.o_pull),
                                                                            b2.at<uint64_t>(wv.o_gpre), wv.npull,
                                                                            wv.run_words, d_elems);
            ::asdm::count_launch();
        }
        if (wv.words) {
            k2_and<<<grid_for(wv.words, G->num_sms), kBlock, 0, s>>>(b2.at<CompDesc>(wv.o_and), b2.at<uint64_t>(wv.o_wpre),
                                                                     wv.nand);
            ::asdm::count_launch();
        }
    }
    ASDM_CUDA(cudaGetLastError());
    auto arena = std::make_shared<CsArena>();
    arena->stream = s;
    {
        std::vector<uint64_t> pos(ntiles + 1, 0);
        std::vector<uint32_t> sizes(nfinal, 0);
        if (ntiles) {
            uint32_t *d_cnt = nullptr, *d_sc = nullptr;
            uint64_t *d_pos = nullptr;
            ASDM_TRY(scr.alloc(&d_cnt, ntiles));
            ASDM_TRY(scr.alloc(&d_pos, ntiles + 1 + (nfinal + 1) / 2));  // positions, then the segments' sizes
            d_sc = reinterpret_cast<uint32_t *>(d_pos + ntiles + 1);
            k3_count<<<(unsigned)ntiles, kBlock, 0, s>>>(b2.at<CompDesc>(o_segs), b2.at<uint64_t>(o_tf), nfinal, d_cnt);
            ::asdm::count_launch();
            ASDM_CUDA(cudaGetLastError());
            ASDM_TRY(scan_exclusive_u32(d_cnt, d_pos, ntiles, true, s));
            uint64_t room = cand_bound;
            if (cand_bound > kCandBound) {
                ASDM_CUDA(cudaMemcpyAsync(&room, d_pos + ntiles, sizeof(uint64_t), cudaMemcpyDeviceToHost, s));
                ASDM_CUDA(cudaStreamSynchronize(s));
            }
            ASDM_TRY(dalloc(&arena->d_cand, room, s));
            k3_write<<<(unsigned)ntiles, kBlock, 0, s>>>(b2.at<CompDesc>(o_segs), b2.at<uint64_t>(o_tf), nfinal, d_pos,
                                                        g.vbl, arena->d_cand, d_sc);
            ::asdm::count_launch();
            ASDM_CUDA(cudaGetLastError());
            std::vector<uint64_t> back(ntiles + 1 + (nfinal + 1) / 2);
            ASDM_CUDA(cudaMemcpyAsync(back.data(), d_pos, back.size() * sizeof(uint64_t), cudaMemcpyDeviceToHost, s));
            ASDM_CUDA(cudaStreamSynchronize(s));
            std::copy(back.begin(), back.begin() + ntiles + 1, pos.begin());
            const uint32_t *sc = reinterpret_cast<const uint32_t *>(back.data() + ntiles + 1);
            for (uint32_t i = 0; i < nfinal; ++i)
                sizes[i] = tile_first[i + 1] > tile_first[i] ? sc[i] : 0;  // a label without vertices has no tile
        }
        std::vector<uint32_t> ncand(nseg, 0);
        std::vector<uint64_t> cbase(nseg, 0);
        for (size_t i = 0; i < seg_ids.size(); ++i) {
            ncand[seg_ids[i]] = sizes[i];
            cbase[seg_ids[i]] = pos[tile_first[i]];
        }
        if (!arena->d_cand) ASDM_TRY(dalloc(&arena->d_cand, 1, s));
        for (QPlan &qp : P) {
            if (qp.empty) continue;
            asdm_cs &cs = *qp.cs;
            bool ok = true;
            for (uint32_t u = 0; u < cs.q.n; ++u) {
                cs.ncand[u] = ncand[qp.seg0 + u];
                cs.cand_base[u] = cbase[qp.seg0 + u];
                ok &= cs.ncand[u] > 0;
            }
            cs.cand_base[cs.q.n] = cs.cand_base[cs.q.n - 1] + cs.ncand[cs.q.n - 1];
            qp.empty = !ok;
        }
    }
    std::vector<EdgeDesc> edges;
    std::vector<uint64_t> item_base{0};
    std::vector<uint32_t> edge_first(Q, 0);
    uint64_t list_bound = 0;  // of all lists: at most |C(u2)| or the largest degree each
    for (uint32_t qi = 0; qi < Q; ++qi) {
        const QPlan &qp = P[qi];
        edge_first[qi] = (uint32_t)edges.size();
        if (qp.empty) continue;
        const asdm_cs &cs = *qp.cs;
        const QueryGraph &q = cs.q;
        for (uint32_t u = 0; u < q.n; ++u)
            for (uint32_t e = q.off[u]; e < q.off[u + 1]; ++e) {
                const uint32_t u2 = q.nbr[e];
                const uint32_t s2 = qp.seg0 + u2;
                edges.push_back(
                    EdgeDesc{arena->d_cand + cs.cand_base[u], (uint32_t)mword[s2], cs.ncand[u], q.lab[u2], 0});
                item_base.push_back(item_base.back() + cs.ncand[u] + 1);
                list_bound += (uint64_t)cs.ncand[u] * std::min(cs.ncand[u2], G->max_deg);
            }
    }
    const uint32_t ne = (uint32_t)edges.size();
    const uint64_t nitems = item_base.back();
    std::vector<uint64_t> estart(ne, 0);
    bool two_scan = false;
    uint64_t total = 0, run_entries = 0;
    if (ne) {
        Blob b3;
        const size_t o_edges = b3.put(edges), o_ib = b3.put(item_base);
        ASDM_TRY(b3.upload(scr));
        const EdgeDesc *d_edges = b3.at<EdgeDesc>(o_edges);
        const uint64_t *d_ib = b3.at<uint64_t>(o_ib);
        uint64_t *d_wpos = nullptr, *d_estart = nullptr;
        uint32_t *d_bad = b1.at<uint32_t>(o_bad);
        ASDM_TRY(scr.alloc(&d_estart, ne));
        ASDM_TRY(dalloc(&arena->d_eoff, nitems, s));
        const unsigned egrid = grid_for(nitems, G->num_sms);
        // One scan of the neighbour runs into a staging buffer of their total
        // length, packed densely after; the exact two-scan form (count, then fill) where that would
        // be too large.  K3 keeps edge-major order: a warp's lanes take
        // consecutive candidates of one edge, whose ascending ids put their
        // adjacency runs side by side in the CSR (grouping by vertex block
        // across edges measured slower).
        uint64_t bound = 0;
        uint32_t *rstart = nullptr;
        uint64_t *d_upos = nullptr;
        // The two scans; the lists get room for `room` entries, 0 for what the first scan counts.
        auto count_then_fill = [&](uint64_t room) {
            ASDM_TRY(scr.alloc(&d_wpos, nitems + 1));
            k3_edges<false><<<egrid, kBlock, 0, s>>>(g, d_edges, cmem, d_ib, ne, arena->d_eoff, nullptr, nullptr,
                                                    d_elems + 1);
            ::asdm::count_launch();
            ASDM_CUDA(cudaGetLastError());
            ASDM_TRY(scan_exclusive_u32(arena->d_eoff, d_wpos, nitems, true, s));
            ASDM_CUDA(cudaMemcpyAsync(&total, d_wpos + nitems, sizeof(uint64_t), cudaMemcpyDeviceToHost, s));
            if (!room) ASDM_CUDA(cudaStreamSynchronize(s));
            ASDM_TRY(dalloc(&arena->d_elist, room ? room : total, s));
            k3_edges<true><<<egrid, kBlock, 0, s>>>(g, d_edges, cmem, d_ib, ne, nullptr, d_wpos, arena->d_elist, nullptr);
            ::asdm::count_launch();
            k3_offsets<<<egrid, kBlock, 0, s>>>(d_ib, ne, d_wpos, arena->d_eoff, d_estart, d_bad);
            ::asdm::count_launch();
            ASDM_CUDA(cudaGetLastError());
            return (int)ASDM_OK;
        };
        // Small groups take the two-scan form too, whose four launches and one
        // readback are quicker than the chunked fill's eight and three
        // (one 8-vertex query on 3,112 vertices: 490 -> 418 us a call).  Up to
        // kListBound possible entries the lists get room for all of them.  A
        // group whose lists could pass the staging cap is not small: the cap
        // decides about it below.
        const uint64_t padded_cap = 1ull << G->tuning.padded_cap_log2;
        const bool small = nitems <= kSmallItems && list_bound <= std::min(kSmallLists, padded_cap);
        if (small) {
            ASDM_TRY(count_then_fill(list_bound > kListBound ? 0 : list_bound));
        } else {
            ASDM_TRY(scr.alloc(&rstart, nitems));
            ASDM_TRY(scr.alloc(&d_upos, nitems + 1));
            k3_bound<<<egrid, kBlock, 0, s>>>(g, d_edges, d_ib, ne, arena->d_eoff, rstart);
            ::asdm::count_launch();
            ASDM_CUDA(cudaGetLastError());
            ASDM_TRY(scan_exclusive_u32(arena->d_eoff, d_upos, nitems, true, s));
            ASDM_CUDA(cudaMemcpyAsync(&bound, d_upos + nitems, sizeof(uint64_t), cudaMemcpyDeviceToHost, s));
            ASDM_CUDA(cudaStreamSynchronize(s));
            // staging buffers of up to 2^padded_cap_log2 entries (default 2^33: 32 GiB)
            two_scan = bound > padded_cap || nitems >= 0xFFFFFF00ull;  // k3_fill numbers items in 32 bits
            if (!two_scan) {
                const uint32_t clog = chunk_log2_for(bound, G->num_sms);
                const uint32_t nchunks = (uint32_t)std::max<uint64_t>(1, (bound + (1ull << clog) - 1) >> clog);
                uint2 *d_chunk = nullptr;  // the chunks' first items
                uint32_t *d_stage = nullptr, *d_chits = nullptr;
                uint64_t *d_cbase = nullptr;
                ASDM_TRY(scr.alloc(&d_stage, (uint64_t)nchunks << clog));
                ASDM_TRY(scr.alloc(&d_chunk, nchunks));
                ASDM_TRY(scr.alloc(&d_chits, nchunks));
                ASDM_TRY(scr.alloc(&d_cbase, (uint64_t)nchunks + 1));
                if (bound == 0) ASDM_CUDA(cudaMemsetAsync(d_chunk, 0, sizeof(uint2), s));
                k3_chunks<<<egrid, kBlock, 0, s>>>(d_ib, ne, d_upos, clog, d_chunk);
                ::asdm::count_launch();
                const unsigned cgrid = grid_for(32ull * nchunks, G->num_sms);  // a warp per chunk
                k3_fill<<<cgrid, kBlock, 0, s>>>(g, d_edges, cmem, d_ib, ne, d_upos, rstart, d_chunk, nchunks, clog,
                                                 arena->d_eoff, d_stage, d_chits);
                ::asdm::count_launch();
                ASDM_CUDA(cudaGetLastError());
                ASDM_TRY(scan_exclusive_u32(d_chits, d_cbase, nchunks, true, s));
                ASDM_CUDA(cudaMemcpyAsync(&total, d_cbase + nchunks, sizeof(uint64_t), cudaMemcpyDeviceToHost, s));
                k3_starts<<<(ne + kBlock - 1) / kBlock, kBlock, 0, s>>>(d_ib, ne, d_upos, nchunks, clog, d_cbase, arena->d_eoff,
                                                                       d_estart);
                ::asdm::count_launch();
                k3_rebase<<<egrid, kBlock, 0, s>>>(d_ib, ne, d_upos, nchunks, clog, d_cbase, d_estart, arena->d_eoff);
                ::asdm::count_launch();
                ASDM_CUDA(cudaStreamSynchronize(s));
                ASDM_TRY(dalloc(&arena->d_elist, total, s));
                k3_pack<<<cgrid, kBlock, 0, s>>>(d_stage, d_chits, d_cbase, nchunks, clog, arena->d_elist);
                ::asdm::count_launch();
                ASDM_CUDA(cudaGetLastError());
                run_entries = bound;
            } else {
                ASDM_TRY(count_then_fill(0));
            }
        }
        uint32_t bad = 0;
        ASDM_CUDA(cudaMemcpyAsync(estart.data(), d_estart, ne * sizeof(uint64_t), cudaMemcpyDeviceToHost, s));
        if (two_scan || small) ASDM_CUDA(cudaMemcpyAsync(&bad, d_bad, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
        ASDM_CUDA(cudaStreamSynchronize(s));
        for (uint32_t e = 0; e < ne && !bad; ++e)
            bad = (e + 1 < ne ? estart[e + 1] : total) - estart[e] > 0xFFFFFFFFull;
        if (bad) return fail(ASDM_ERR_INVALID, "a candidate-edge list exceeds 2^32 entries");
    }
    unsigned long long elems[2] = {0, 0};
    ASDM_CUDA(cudaMemcpyAsync(elems, d_elems, 2 * sizeof(unsigned long long), cudaMemcpyDeviceToHost, s));
    ASDM_CUDA(cudaEventRecord(ev1, s));
    ASDM_CUDA(cudaStreamSynchronize(s));
    float ms = 0.f;
    cudaEventElapsedTime(&ms, ev0, ev1);
    cudaEventDestroy(ev0);
    cudaEventDestroy(ev1);
    // K1 reads 8 bytes per vertex of the label of each distinct query-vertex
    // signature (and copies F words for the repeats); K2 and K3 read one rank
    // per scanned neighbour; compaction reads the bitsets it ANDs; K3 writes
    // the candidate-edge lists and their offsets (4 bytes per entry)
    const uint64_t bytes = 8ull * seg.back() + 8ull * copied_words + 4ull * (elems[0] + elems[1] + run_entries) +
                           4ull * bit_words_read + 4ull * total + 4ull * nitems;
    for (uint32_t qi = 0; qi < Q; ++qi) {
        QPlan &qp = P[qi];
        asdm_cs &cs = *qp.cs;
        cs.build_ms = ms / Q;
        cs.build_bytes = bytes / Q;
        cs.build_flags = (two_scan ? ASDM_CS_TWO_SCAN : 0u) | (g.lab_pos ? ASDM_CS_LABEL_RUNS : 0u);
        cs.arena = arena;
        cs.d_cand = arena->d_cand;
        cs.d_eoff = arena->d_eoff;
        cs.d_elist = arena->d_elist;
        if (qp.empty) {
            cs.nonempty = false;
            continue;
        }
        cs.nonempty = true;
        const QueryGraph &q = cs.q;
        const uint32_t nq_e = q.off[q.n];
        cs.eoff_base.assign(nq_e, 0);
        cs.elist_base.assign(nq_e, 0);
        cs.etotal.assign(nq_e, 0);
        for (uint32_t k = 0; k < nq_e; ++k) {
            const uint32_t e = edge_first[qi] + k;
            cs.eoff_base[k] = item_base[e];
            cs.elist_base[k] = estart[e];
            const uint64_t end = (e + 1 < ne) ? estart[e + 1] : total;
            cs.etotal[k] = end - estart[e];
        }
    }
    return ASDM_OK;
}

}  // namespace asdm

using namespace asdm;

extern "C" int asdm_candidate_space(asdm_graph *g, const uint32_t *q_offsets, const uint32_t *q_nbrs,
                                    const uint32_t *q_labels, uint32_t q_n, asdm_cs **out, int *nonempty) {
    clear_error();
    if (!g || !out) return fail(ASDM_ERR_INVALID, "null argument");
    auto cs = std::make_unique<asdm_cs>();
    cs->g = g;
    ASDM_TRY(make_query(q_offsets, q_nbrs, q_labels, q_n, cs->q));
    int rc = build_batch({cs.get()});
    if (rc != ASDM_OK) {
        cs.reset();
        cudaStreamSynchronize(g->stream);
        return rc;
    }
    if (nonempty) *nonempty = cs->nonempty ? 1 : 0;
    *out = cs.release();
    return ASDM_OK;
}

extern "C" int asdm_cs_sizes(const asdm_cs *cs, uint32_t *sizes) {
    if (!cs || !sizes) return fail(ASDM_ERR_INVALID, "null argument");
    for (uint32_t u = 0; u < cs->q.n; ++u) sizes[u] = cs->ncand.empty() ? 0 : cs->ncand[u];
    return ASDM_OK;
}

extern "C" int asdm_cs_read(const asdm_cs *cs, uint32_t u, uint32_t *out, uint32_t capacity) {
    if (!cs || !out) return fail(ASDM_ERR_INVALID, "null argument");
    if (u >= cs->q.n) return fail(ASDM_ERR_INVALID, "query vertex %u out of range", u);
    const uint32_t n = cs->ncand.empty() ? 0 : cs->ncand[u];
    if (n > capacity) return fail(ASDM_ERR_CAPACITY, "candidate set of %u has %u entries", u, n);
    if (n == 0) return ASDM_OK;
    ASDM_CUDA(cudaMemcpyAsync(out, cs->d_cand + cs->cand_base[u], n * sizeof(uint32_t), cudaMemcpyDeviceToHost,
                              cs->g->stream));
    ASDM_CUDA(cudaStreamSynchronize(cs->g->stream));
    return ASDM_OK;
}

extern "C" int asdm_cs_read_edges(const asdm_cs *cs, uint32_t u, uint32_t u2, uint32_t *offsets, uint32_t *vertices,
                                  uint64_t capacity, uint64_t *total) {
    if (!cs || !offsets) return fail(ASDM_ERR_INVALID, "null argument");
    if (u >= cs->q.n || u2 >= cs->q.n) return fail(ASDM_ERR_INVALID, "query vertex out of range");
    const int k = cs->q.slot(u, u2);
    if (k < 0) return fail(ASDM_ERR_INVALID, "(%u, %u) is not a query edge", u, u2);
    if (!cs->nonempty) return fail(ASDM_ERR_INVALID, "candidate space is empty");
    const uint32_t e = cs->q.off[u] + (uint32_t)k;
    const uint64_t cnt = cs->etotal[e];
    if (total) *total = cnt;
    if (cnt > capacity) return fail(ASDM_ERR_CAPACITY, "edge list has %llu entries", (unsigned long long)cnt);
    cudaStream_t s = cs->g->stream;
    const uint32_t nu = cs->ncand[u], nu2 = cs->ncand[u2];
    ASDM_CUDA(cudaMemcpyAsync(offsets, cs->d_eoff + cs->eoff_base[e], (nu + 1) * sizeof(uint32_t),
                              cudaMemcpyDeviceToHost, s));
    std::vector<uint32_t> idx(cnt), c2(nu2);
    if (cnt) ASDM_CUDA(cudaMemcpyAsync(idx.data(), cs->d_elist + cs->elist_base[e], cnt * sizeof(uint32_t),
                                       cudaMemcpyDeviceToHost, s));
    ASDM_CUDA(cudaMemcpyAsync(c2.data(), cs->d_cand + cs->cand_base[u2], nu2 * sizeof(uint32_t),
                              cudaMemcpyDeviceToHost, s));
    ASDM_CUDA(cudaStreamSynchronize(s));
    if (vertices)
        for (uint64_t i = 0; i < cnt; ++i) vertices[i] = c2[idx[i]];
    return ASDM_OK;
}

extern "C" int asdm_cs_free(asdm_cs *cs) {
    if (!cs) return ASDM_OK;
    cudaStream_t s = cs->g->stream;
    delete cs;  // the group's arena is freed with its last candidate space
    cudaStreamSynchronize(s);
    return ASDM_OK;
}
