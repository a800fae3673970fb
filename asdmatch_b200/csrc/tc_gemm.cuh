// BF16 x BF16 -> FP32 tile GEMM on the 5th-generation tensor cores (tcgen05).
//
//   D[m][n] = sum_k A(m, k) * B(n, k)      one 128 x 128 output tile per CTA
//
// A and B are read from global memory through caller-supplied strides, 64
// K-elements at a time, into shared memory in the canonical K-major,
// no-swizzle core-matrix layout (8 rows x 16 bytes per core matrix), and
// multiplied by tcgen05.mma issued from one thread, M=128 N=128 K=16 per
// instruction, accumulating in tensor memory.  An operand whose K runs along
// memory is copied with 16-byte cp.async, one whose rows do is loaded 16 bytes
// at a time and transposed in registers, 8 x 8 elements a thread; element by
// element only where alignment or a ragged edge asks for it.  kStages chunks
// of shared memory are in rotation: chunks are fetched kStages - 1 ahead of
// the tensor cores (element-wise, unbuffered staging took 10 us a chunk: a
// forward product of 4,600 nodes 97 us).  With splits, the K chunks are
// divided among grid.z CTAs, whose fp32 partial products split_sum adds in
// order: the weight gradients' K is the node count, which would otherwise
// leave two CTAs working.
// tcgen05.commit arrives on the stage's mbarrier, waited for (bounded) before
// the stage is refilled or the accumulator is read back with tcgen05.ld.
// 128 threads (4 warps): warp w owns TMEM lanes 32w..32w+31, i.e. output rows
// 32w..32w+31 of the tile.
#pragma once

#include <cuda_bf16.h>
#include <cstdint>

#include "mma_steps.h"

namespace asdm {
namespace tc {

constexpr int kTileM = 128, kTileN = 128, kChunkK = 64;
constexpr int kThreads = 128;
constexpr uint32_t kTmemCols = 128;
constexpr uint32_t kWaitSpins = 1u << 22;
constexpr int kStages = 3;
// Core matrices lie kCore bytes apart along the rows (16 more than their 128,
// so that stores of one row of neighbouring matrices fall into different
// banks) and kGroup apart along K.
constexpr int kCore = 144, kGroup = (kTileM / 8) * kCore, kOperand = (kChunkK / 8) * kGroup;
// stages, mbarriers, TMEM address.  At most two CTAs share an SM: 2 x 128 TMEM
// columns never exceed the SM's 512, so tcgen05.alloc never has to wait.
constexpr int kSmemBytes = kStages * 2 * kOperand + 64;

// Operand view: element (r, k) at ptr[r * sr + k * sk]; rows >= rows_valid
// and k >= K read as zero.
struct Operand {
    const __nv_bfloat16 *ptr;
    long long sr, sk;
    int rows_valid;
};

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// tcgen05 shared-memory matrix descriptor, SWIZZLE_NONE, version 1.
__device__ __forceinline__ uint64_t make_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFF) >> 4);
    d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
    d |= 1ull << 46;  // descriptor version for sm_100
    return d;           // base offset 0, absolute-LBO mode off, layout type 0 (no swizzle)
}

// Instruction descriptor, kind::f16: D=F32, A=B=BF16, both K-major, M=128, N=128.
__host__ __device__ constexpr uint32_t idesc_bf16_f32() {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kTileN >> 3) << 17) | ((uint32_t)(kTileM >> 4) << 24);
}

// Byte offset of element (row r, k) of a staged chunk: core (row group, k
// group) at kGroup * (k / 8) + kCore * (r / 8), row r of the group at +16 r.
__device__ __forceinline__ int staged_at(int r, int k) { return (k >> 3) * kGroup + (r >> 3) * kCore + (r & 7) * 16 + (k & 7) * 2; }

__device__ __forceinline__ void stage_core_row(uint8_t *dst, const Operand &op, int gr, int gk, int K) {
    __nv_bfloat16 *d = reinterpret_cast<__nv_bfloat16 *>(dst);
#pragma unroll
    for (int j = 0; j < 8; ++j)
        d[j] = gr < op.rows_valid && gk + j < K ? op.ptr[(long long)gr * op.sr + (long long)(gk + j) * op.sk]
                                                : __float2bfloat16(0.f);
}

// Stage rows [r0, r0+128) x k [k0, k0+64) of an operand.
__device__ __forceinline__ void stage(uint8_t *dst, const Operand &op, int r0, int k0, int K) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (op.sr == 1 && op.sk % 8 == 0 && (reinterpret_cast<uintptr_t>(op.ptr) & 15) == 0) {
        // rows along memory: thread (k group, row group) loads 8 rows of 8 k and transposes them
        const int rg = threadIdx.x & 15, kg = threadIdx.x >> 4, gr = r0 + 8 * rg, gk = k0 + 8 * kg;
        uint8_t *d = dst + kg * kGroup + rg * kCore;
        if (gr + 8 <= op.rows_valid) {
            uint32_t w[8][4];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                uint4 v = make_uint4(0, 0, 0, 0);
                if (gk + j < K) v = *reinterpret_cast<const uint4 *>(op.ptr + gr + (long long)(gk + j) * op.sk);
                w[j][0] = v.x; w[j][1] = v.y; w[j][2] = v.z; w[j][3] = v.w;
            }
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                uint32_t o[4];
#pragma unroll
                for (int j = 0; j < 4; ++j)  // k 2j and 2j + 1 of row r
                    o[j] = __byte_perm(w[2 * j][r >> 1], w[2 * j + 1][r >> 1], (r & 1) ? 0x7632 : 0x5410);
                *reinterpret_cast<uint4 *>(d + 16 * r) = make_uint4(o[0], o[1], o[2], o[3]);
            }
        } else {
            for (int r = 0; r < 8; ++r) stage_core_row(d + 16 * r, op, gr + r, gk, K);
        }
        return;
    }
    const bool vec = op.sk == 1 && op.sr % 8 == 0 && (reinterpret_cast<uintptr_t>(op.ptr) & 15) == 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        // a warp copies 8 rows x 4 k groups: whole core matrices
        const int c = i * 4 + warp, r = (c >> 1) * 8 + (lane & 7), k = ((c & 1) * 4 + (lane >> 3)) * 8;
        uint8_t *d = dst + staged_at(r, k);
        const int gr = r0 + r, gk = k0 + k;
        const bool in = gr < op.rows_valid && gk < K;
        if (vec && (!in || gk + 8 <= K)) {
            const __nv_bfloat16 *src = in ? op.ptr + (long long)gr * op.sr + gk : op.ptr;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(d)), "l"(src), "r"(in ? 16 : 0));
        } else {
            stage_core_row(d, op, gr, gk, K);
        }
    }
}

// Waits (bounded) for the mbarrier's phase.
__device__ __forceinline__ bool wait_phase(uint64_t *mbar, uint32_t parity) {
    uint32_t done = 0;
    for (uint32_t it = 0; it < kWaitSpins && !done; ++it) {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done)
            : "r"(smem_u32(mbar)), "r"(parity));
    }
    return done != 0;
}

// Computes one 128x128 tile of the K chunks [c0, c1) into C (fp32, row-major
// with stride ldc), rows >= m_valid / cols >= n_valid not written.  `err` gets 1 if a wait on
// the tensor cores ran out of its bound (the tile is then not written).
__device__ void gemm_tile(const Operand &A, const Operand &B, int K, int c0, int c1, int m0, int n0, float *C,
                          long long ldc, int m_valid, int n_valid, const float *bias, bool relu, unsigned int *err) {
    extern __shared__ __align__(1024) uint8_t smem[];
    uint64_t *mbar = reinterpret_cast<uint64_t *>(smem + kStages * 2 * kOperand);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(mbar + kStages);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(kTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (threadIdx.x < kStages) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(mbar + threadIdx.x)));
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = *tmem_slot;

    const int nc = c1 - c0;
    const uint32_t idesc = idesc_bf16_f32();
    auto fetch = [&](int i) {  // chunk i of this CTA into its stage (an empty group past the end)
        if (i < nc) {
            uint8_t *d = smem + (i % kStages) * 2 * kOperand;
            stage(d, A, m0, (c0 + i) * kChunkK, K);
            stage(d + kOperand, B, n0, (c0 + i) * kChunkK, K);
        }
        asm volatile("cp.async.commit_group;");
    };
    auto issue = [&](int i) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2));  // chunk i has landed
        // make the generic-proxy smem writes visible to the tensor cores
        asm volatile("fence.proxy.async.shared::cta;");
        __syncthreads();
        if (threadIdx.x == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;");
            const uint32_t sa = smem_u32(smem + (i % kStages) * 2 * kOperand), sb = sa + kOperand;
            for (int s = 0; s < kChunkK / 16; ++s) {
                // K slice s: k groups 2s, 2s+1
                const uint64_t da = make_desc(sa + s * 2 * kGroup, kGroup, kCore);
                const uint64_t db = make_desc(sb + s * 2 * kGroup, kGroup, kCore);
                const uint32_t accumulate = (i > 0 || s > 0) ? 1u : 0u;
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "setp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n"
                    :
                    : "r"(tmem), "l"(da), "l"(db), "r"(idesc), "r"(accumulate), "r"(0u), "r"(0u), "r"(0u), "r"(0u));
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                smem_u32(mbar + i % kStages)));
        }
    };
    // chunk i's commit covers the products of every chunk before it
    auto wait = [&](int i) { return wait_phase(mbar + i % kStages, (uint32_t)(i / kStages) & 1u); };
    const bool ok = run_chunks<kStages>(nc, fetch, issue, wait, [](bool x) { return __syncthreads_and(x) != 0; });
    asm volatile("cp.async.wait_all;");
    asm volatile("tcgen05.fence::after_thread_sync;");
    if (ok) {
        const int row = m0 + warp * 32 + lane;
        const bool vec = (ldc & 3) == 0 && (n_valid & 3) == 0 && (reinterpret_cast<uintptr_t>(C) & 15) == 0;
        for (int c = 0; c < kTileN; c += 16) {
            uint32_t r[16];
            asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
                         "%14, %15}, [%16];\n"
                         : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                           "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                         : "r"(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c));
            asm volatile("tcgen05.wait::ld.sync.aligned;");
            if (row >= m_valid) continue;
#pragma unroll
            for (int j = 0; j < 16; j += 4) {
                const int col = n0 + c + j;
                float v[4];
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    v[t] = nc > 0 ? __uint_as_float(r[j + t]) : 0.f;  // no chunks: nothing was accumulated
                    if (bias && col + t < n_valid) v[t] += bias[col + t];
                    if (relu) v[t] = fmaxf(v[t], 0.f);
                }
                float *dst = C + (long long)row * ldc + col;
                if (vec && col < n_valid) {
                    *reinterpret_cast<float4 *>(dst) = make_float4(v[0], v[1], v[2], v[3]);
                } else {
#pragma unroll
                    for (int t = 0; t < 4; ++t)
                        if (col + t < n_valid) dst[t] = v[t];
                }
            }
        }
    } else {
        // a wait ran out; the products in flight had one more bounded wait (run_chunks)
        if (threadIdx.x == 0) atomicExch(err, 1u);
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols));
}

// grid (ceil(M/128), ceil(N/128), splits); dynamic shared memory kSmemBytes.
// With splits > 1, split z writes its partial product to C + z * M * ldc.
__global__ void __launch_bounds__(kThreads) gemm_kernel(Operand A, Operand B, int M, int N, int K, float *C, long long ldc,
                                                        const float *bias, int relu, unsigned int *err) {
    const int chunks = (K + kChunkK - 1) / kChunkK, per = (chunks + (int)gridDim.z - 1) / (int)gridDim.z;
    const int c0 = min(chunks, (int)blockIdx.z * per), c1 = min(chunks, c0 + per);
    gemm_tile(A, B, K, c0, c1, blockIdx.x * kTileM, blockIdx.y * kTileN, C + (long long)blockIdx.z * M * ldc, ldc, M, N,
              bias, relu != 0, err);
}

// out[i] = sum of the splits' partial products, in order.
__global__ void split_sum(const float *__restrict__ part, int splits, long long n, float *__restrict__ out) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        float s = 0.f;
#pragma unroll 8
        for (int z = 0; z < splits; ++z) s += part[z * n + i];
        out[i] = s;
    }
}

}  // namespace tc
}  // namespace asdm
