// mlp.cu -- dense layers of the brick-mode selector on the 5th-generation tensor cores.
//
// One GEMM form serves the forward and the backward pass:
//     C[M][N] = epilogue(A[M][K] . B[N][K]^T)
// with A and B bf16, row-major with K contiguous ("K-major"), fp32 accumulation
// in tensor memory, and an epilogue that adds a bias, applies ReLU or the ReLU
// gradient mask, and writes fp32 and/or bf16, plain or transposed.
//
// Per CTA: one 128 x N tile (N <= 64, or 256 in place, a multiple of 16), 128 threads.  The selector's
// layers are small (2048 x 256 x 256 at the training batch), so tiles are narrow, to
// spread over the SMs.  K runs in chunks of 64 through four stages of shared memory in the
// canonical no-swizzle K-major layout (8-row x 16-byte core matrices; core matrix (row
// group g, column group c) at (g * 8 + c) * 128 bytes, so the K-adjacent core matrices are
// 128 bytes apart and the row-adjacent ones 1024).  One thread issues four tcgen05.mma
// (M=128, N, K=16) per chunk with the accumulator in tensor memory and commits them to the
// stage's mbarrier.  The network's own operands lie in global memory in that layout, chunk
// after chunk (tiled_at), so that the same thread fills a stage with one bulk copy per
// operand and nothing else of the block takes part; row-major operands (csv_gemm_bf16) are
// copied by all threads with cp.async, a block barrier per chunk.  (A product over 2048
// rows: 30 us row-major, 20 us tiled.)  The epilogue reads the accumulator with tcgen05.ld
// (warp w owns lanes 32w..32w+31 = rows) and applies the fused ops.  An output's products
// are added in the order of K whatever the tile, so results do not depend on it.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>

#include "csv_internal.h"

namespace csv {
namespace {

constexpr uint32_t kGemmThreads = 128;
constexpr uint32_t kKChunk = 64;               // bf16 elements per row per chunk (128 bytes)
constexpr uint32_t kTileN = 64;                // columns per CTA at most
constexpr uint32_t kTileWide = 256;            // the same in the wide form, which stages kTileN of them at a time
constexpr uint32_t kStages = 4;
constexpr uint32_t kTileA = 128 * kKChunk * 2; // 16 KB
constexpr uint32_t kTileB = kTileN * kKChunk * 2;  // 8 KB
constexpr uint32_t kWaitLimit = 1u << 24;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
    // start address, leading byte offset (K-adjacent core matrices), stride byte
    // offset (row-adjacent core matrices), descriptor version 1, no swizzle
    const uint64_t lbo = 128, sbo = 1024;
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((lbo >> 4) << 16) | ((sbo >> 4) << 32) | (1ull << 46);
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}

__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void expect_bytes(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem, uint64_t ad, uint64_t bd, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
        "l"(ad), "l"(bd), "r"(idesc), "r"(acc)
        : "memory");
}

__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
    for (uint32_t it = 0; it < kWaitLimit; ++it) {
        uint32_t done;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t v[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
    const uint32_t lo = __bfloat16_as_ushort(__float2bfloat16_rn(a));
    const uint32_t hi = __bfloat16_as_ushort(__float2bfloat16_rn(b));
    return lo | (hi << 16);
}

__device__ __forceinline__ bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

// Rows [r0, r0 + n) of a K-major operand, 64 K elements from k0 on, into core matrices (n
// a multiple of 8).  Eight lanes read 32 bytes of four rows each.
__device__ __forceinline__ void load_operand(uint32_t dst, const __nv_bfloat16* src, uint32_t K, uint32_t r0, uint32_t n,
                                             uint32_t k0) {
    for (uint32_t u = threadIdx.x; u < n * 8u; u += kGemmThreads) {
        const uint32_t r = ((u >> 1) & 7u) + 8 * (u >> 6), kb = (u & 1u) | ((u >> 3) & 6u);
        cp_async16(dst + ((r >> 3) * 8 + kb) * 128 + (r & 7u) * 16, src + (size_t)(r0 + r) * K + k0 + kb * 8);
    }
}

// Softmax cross-entropy of the mode head (logits 0..11) and the table head (12..27) of one
// row against its label: g = (softmax - onehot) / n; returns the row's loss / n.
__device__ __forceinline__ float loss_grad_row(const float (&z)[32], uint32_t label, uint32_t n, float (&g)[32]) {
    float l = 0.0f;
#pragma unroll
    for (int head = 0; head < 2; ++head) {
        constexpr int first[2] = {0, 12}, cnt[2] = {12, 16};
        const int y = head ? label >> 4 : label & 15u;
        float mx = -INFINITY;
#pragma unroll
        for (int k = 0; k < 16; ++k)
            if (k < cnt[head]) mx = fmaxf(mx, z[first[head] + k]);
        float se = 0.0f, zy = 0.0f;
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            if (k < cnt[head]) {
                g[first[head] + k] = expf(z[first[head] + k] - mx);
                se += g[first[head] + k];
            }
            if (k == y) zy = z[first[head] + k];
        }
#pragma unroll
        for (int k = 0; k < 16; ++k)
            if (k < cnt[head]) g[first[head] + k] = (g[first[head] + k] / se - (k == y ? 1.0f : 0.0f)) / (float)n;
        l += logf(se) + mx - zy;
    }
    return l / (float)n;
}

// Up to two products in one launch: the first n_first blocks are the first one's.
// Bound by latency: a layer of the training batch is a few tiles of work, and a product
// over the rows one chain of chunks per output.  Tiles of 16 columns for the latter spread
// it over four times the SMs; a split of the chain would be shorter yet, but its partial
// sums round apart from the single accumulation's (3.6e-5 of the gradient at 14,826 rows).
// Measured (B200, a gradient step of 2048 rows; 128 x 256 tiles whose 64-wide chunks were
// loaded and multiplied in turn, products over the rows on 2 CTAs, bias sums by one block
// each): 0.87 -> 0.105 ms of kernels (0.7 us at the bf16 rate); a 2048 x 256 x 256 layer
// 74 -> 9.5 us, the 256 x 256 product over the rows 171 -> 20 us beside the next layer's.
template <bool TILED, bool WIDE>
__global__ void __launch_bounds__(kGemmThreads) gemm_bf16_kernel(GemmArgs G0, GemmArgs G1, uint32_t n_first) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t bars[kStages], full[kStages];  // a stage's products done; its copies landed (TILED)
    __shared__ uint32_t s_ok;
    __shared__ uint32_t tmem_base;
    const bool second = blockIdx.x >= n_first;
    const GemmArgs& G = second ? G1 : G0;
    const uint32_t blk = second ? blockIdx.x - n_first : blockIdx.x;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    const uint32_t mt = G.M / 128u;
    const uint32_t m0 = (blk % mt) * 128u, n0 = (blk / mt) * G.tile_n;
    const uint32_t N = min(G.tile_n, G.N - n0);
    const uint32_t ncols = N <= 32 ? 32u : (!WIDE || N <= 64 ? 64u : (N <= 128 ? 128u : 256u));
    const uint32_t sA = smem_u32(smem), sB = sA + kStages * kTileA;
    if (tid == 0) {
        for (uint32_t s = 0; s < kStages; ++s) {
            mbar_init(smem_u32(&bars[s]), 1);
            mbar_init(smem_u32(&full[s]), 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                     "r"(ncols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base;
    const uint32_t chunks = G.K / kKChunk;
    auto done = [&](uint32_t c) { return mbar_wait(smem_u32(&bars[c % kStages]), (c / kStages) & 1u); };
    // stage c's products into columns [col, col + n) (first: they start a sum)
    auto multiply = [&](uint32_t c, uint32_t col, uint32_t n, bool first) {
        // M = 128, N = n, bf16 x bf16 -> f32, both operands K-major
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((n >> 3) << 17) | ((128u >> 4) << 24);
#pragma unroll
        for (uint32_t s = 0; s < kKChunk / 16; ++s)
            mma_bf16(tmem + col, smem_desc(sA + (c % kStages) * kTileA + s * 256u),
                     smem_desc(sB + (c % kStages) * kTileB + s * 256u), idesc, (!first || s > 0) ? 1u : 0u);
        mma_commit(smem_u32(&bars[c % kStages]));
    };
    bool ok = true;
    if (TILED) {
        if (tid == 0) {
            auto landed = [&](uint32_t c) { return mbar_wait(smem_u32(&full[c % kStages]), (c / kStages) & 1u); };
            auto load = [&](uint32_t c) {
                const uint32_t s = c % kStages, bar = smem_u32(&full[s]);
                expect_bytes(bar, kTileA + N * kKChunk * 2);
                bulk_g2s(sA + s * kTileA, G.A + tiled_at(G.M, m0, c * kKChunk), kTileA, bar);
                bulk_g2s(sB + s * kTileB, G.B + tiled_at(G.N, n0, c * kKChunk), N * kKChunk * 2, bar);
            };
            uint32_t issued = 0, waited = 0;
            for (; issued < min(kStages, chunks); ++issued) load(issued);
            for (uint32_t c = 0; c < chunks && ok; ++c) {
                ok = landed(c);
                waited = c + 1;
                if (!ok) break;
                multiply(c, 0, N, c == 0);
                // the stage before this one is filled again once its products are done
                if (c > 0 && issued < chunks) {
                    ok = done(c - 1);
                    if (ok) load(issued++);
                }
            }
            if (ok) ok = done(chunks - 1);
            for (; waited < issued; ++waited) landed(waited);  // (after a failure: no copy in flight at the exit)
            s_ok = ok ? 1u : 0u;
        }
        __syncthreads();
        ok = s_ok != 0;
    } else {
        // a step is a chunk of K; WIDE: of 64 columns, all of K for these before the next ones
        const uint32_t steps = WIDE ? (N + kTileN - 1) / kTileN * chunks : chunks;
        auto col = [&](uint32_t c) { return WIDE ? c / chunks * kTileN : 0u; };
        auto chunk = [&](uint32_t c) { return WIDE ? c % chunks : c; };
        auto load = [&](uint32_t c) {  // step c's operands into its stage; a group of copies either way
            if (c < steps) {
                load_operand(sA + (c % kStages) * kTileA, G.A, G.K, m0, 128u, chunk(c) * kKChunk);
                load_operand(sB + (c % kStages) * kTileB, G.B, G.K, n0 + col(c), WIDE ? min(N - col(c), kTileN) : N,
                             chunk(c) * kKChunk);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        for (uint32_t c = 0; c + 1 < kStages; ++c) load(c);
        for (uint32_t c = 0; c < steps; ++c) {
            asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            if (!(ok = __syncthreads_and(ok))) break;  // one decision for the whole block
            if (tid == 0) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                multiply(c, col(c), WIDE ? min(N - col(c), kTileN) : N, chunk(c) == 0);
            }
            if (c > 0) ok = done(c - 1);
            if (ok) load(c + kStages - 1);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        ok = __syncthreads_and(ok && done(steps - 1)) != 0;
    }
    if (!ok && tid == 0 && G.err) atomicExch(G.err, 1u);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t row = m0 + warp * 32u + lane, taddr = tmem + ((warp * 32u) << 16);
    if (ok && G.label) {  // the logits (N = 32): the loss and its gradient
        float z[32], g[32];
        uint32_t v[32];
        tmem_ld16(taddr, v);
        tmem_ld16(taddr + 16, v + 16);
#pragma unroll
        for (uint32_t j = 0; j < 32; ++j) {
            z[j] = __uint_as_float(v[j]) + G.bias[j];
            g[j] = 0.0f;
        }
        float l = 0.0f;
        if (row < G.n_rows) l = loss_grad_row(z, G.label[row], G.n_rows, g);
        for (int o = 16; o > 0; o >>= 1) l += __shfl_down_sync(0xffffffffu, l, o);
        if (lane == 0) atomicAdd(G.loss, l);
        // dZ [rows][64], zero beyond the logits, and its transpose [32][rows], tiled
#pragma unroll
        for (uint32_t q = 0; q < 8; ++q)
            *reinterpret_cast<uint4*>(G.Cb + tiled_at(G.M, row, 8 * q)) =
                q < 4 ? make_uint4(pack_bf16(g[8 * q], g[8 * q + 1]), pack_bf16(g[8 * q + 2], g[8 * q + 3]),
                                   pack_bf16(g[8 * q + 4], g[8 * q + 5]), pack_bf16(g[8 * q + 6], g[8 * q + 7]))
                      : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (uint32_t j = 0; j < 32; ++j) G.CbT[tiled_at(32, j, row)] = __float2bfloat16_rn(g[j]);
    } else if (ok) {
        float *C = G.C, *CT = G.CT;
        // (rows of N = 16 k values: 16-byte pieces when the arrays start on one)
        const bool vec_c = aligned16(C), vec_cb = aligned16(G.Cb), vec_mask = aligned16(G.mask);
        for (uint32_t j0 = 0; j0 < N; j0 += 16) {
            uint32_t v[16];
            tmem_ld16(taddr + j0, v);
            // two runs of eight columns, 16 bytes each: side by side, or in two core matrices
            const size_t at = TILED ? tiled_at(G.M, row, n0 + j0) : (size_t)row * G.N + n0 + j0;
            const uint32_t next8 = TILED ? 64u : 8u;
            float x[16];
#pragma unroll
            for (uint32_t j = 0; j < 16; ++j) {
                x[j] = __uint_as_float(v[j]);
                if (G.bias) x[j] += G.bias[n0 + j0 + j];
                if (G.relu) x[j] = fmaxf(x[j], 0.0f);
            }
            if (G.mask) {
                __nv_bfloat16 m[16];
                if (TILED || vec_mask) {
                    reinterpret_cast<uint4*>(m)[0] = *reinterpret_cast<const uint4*>(G.mask + at);
                    reinterpret_cast<uint4*>(m)[1] = *reinterpret_cast<const uint4*>(G.mask + at + next8);
                } else {
#pragma unroll
                    for (uint32_t j = 0; j < 16; ++j) m[j] = G.mask[at + j];
                }
#pragma unroll
                for (uint32_t j = 0; j < 16; ++j)
                    if (!(__bfloat162float(m[j]) > 0.0f)) x[j] = 0.0f;
            }
            if (C) {  // (row-major either way)
                float* o = C + (size_t)row * G.N + n0 + j0;
                if (vec_c) {
#pragma unroll
                    for (uint32_t q = 0; q < 4; ++q)
                        reinterpret_cast<float4*>(o)[q] =
                            make_float4(x[4 * q], x[4 * q + 1], x[4 * q + 2], x[4 * q + 3]);
                } else {
#pragma unroll
                    for (uint32_t j = 0; j < 16; ++j) o[j] = x[j];
                }
            }
            if (G.Cb) {
                if (TILED || vec_cb) {
#pragma unroll
                    for (uint32_t q = 0; q < 2; ++q)
                        *reinterpret_cast<uint4*>(G.Cb + at + q * next8) =
                            make_uint4(pack_bf16(x[8 * q], x[8 * q + 1]), pack_bf16(x[8 * q + 2], x[8 * q + 3]),
                                       pack_bf16(x[8 * q + 4], x[8 * q + 5]), pack_bf16(x[8 * q + 6], x[8 * q + 7]));
                } else {
#pragma unroll
                    for (uint32_t j = 0; j < 16; ++j) G.Cb[at + j] = __float2bfloat16_rn(x[j]);
                }
            }
            if (G.CbT)
#pragma unroll
                for (uint32_t j = 0; j < 16; ++j)
                    G.CbT[TILED ? tiled_at(G.N, n0 + j0 + j, row) : (size_t)(n0 + j0 + j) * G.M + row] =
                        __float2bfloat16_rn(x[j]);
            if (CT)
#pragma unroll
                for (uint32_t j = 0; j < 16; ++j) CT[(size_t)(n0 + j0 + j) * G.M + row] = x[j];
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncols) : "memory");
}

// ------------------------------------------------------------ fused inference
// The selector's whole forward pass for 128 rows at a time, persistent (one CTA
// per SM, all 512 tensor-memory columns), activations never leaving the SM:
//   X (bf16, features padded to 64) -> acc1 = X W1^T (TMEM cols 0..255)
//   H1 = bf16(relu(acc1 + b1))      -> shared memory, the next A operand
//   acc2 = H1 W2^T (TMEM cols 256..511), W2 streamed from L2 in four 32 KB
//   K-chunks through a two-slot ring of bulk copies (it does not fit beside
//   the rest), H2 = bf16(relu(acc2 + b2)) -> shared memory
//   acc3 = H2 W3^T (TMEM cols 0..31), logits = acc3 + b3, argmax per head.
// A layer's products are added in the K order of the layer-by-layer GEMMs (whose tiles
// are narrower, which changes no sum), so the logits are those of gemm_bf16_kernel's
// three launches.
// Weights come pre-tiled in the no-swizzle K-major core-matrix layout, so that
// each K-chunk is one contiguous bulk copy: K-chunks of 64, each N/8 x 8 core matrices
// of 8 rows x 16 bytes, core (g, c) at (g * 8 + c) * 128 bytes.
constexpr uint32_t kInferThreads = 128;
constexpr uint32_t kHidN = 256, kInN = 64, kOutN = 32;
constexpr uint32_t kSelModes = 12, kSelTables = 16;  // the two heads: logits 0..11 and 12..27
constexpr uint32_t kChunkW2 = kHidN * kKChunk * 2;   // 32 KB
constexpr uint32_t kChunkW3 = kOutN * kKChunk * 2;   // 4 KB
constexpr uint32_t kChunkH = 128 * kKChunk * 2;      // 16 KB
constexpr uint32_t kOffW1 = 0;                       // 32 KB
constexpr uint32_t kOffW3 = kOffW1 + kHidN * kInN * 2;  // 16 KB (4 chunks)
constexpr uint32_t kOffH = kOffW3 + 4 * kChunkW3;       // 64 KB (4 chunks); chunk 0 holds X first
constexpr uint32_t kOffRing = kOffH + 4 * kChunkH;      // 2 x 32 KB
constexpr uint32_t kOffBias = kOffRing + 2 * kChunkW2;  // b1, b2, b3 (fp32)
constexpr uint32_t kInferSmem = kOffBias + (2 * kHidN + kOutN) * 4;

struct InferArgs {
    const float* feat;          // [count][32]
    uint32_t count;
    const __nv_bfloat16* W1t;   // tiled [256][64]
    const __nv_bfloat16* W2t;   // tiled [256][256]: four 32 KB chunks
    const __nv_bfloat16* W3t;   // tiled [32][256]: four 4 KB chunks
    const float *b1, *b2, *b3;
    float* logits;              // [count][32] or null
    uint8_t* sel;               // [count] or null: argmax(0..11) | argmax(12..27) << 4
    uint32_t* err;
};

// (row r, K element k) of a 128-row A operand held as 64-wide K-chunks of core matrices
__device__ __forceinline__ uint32_t a_off(uint32_t r, uint32_t k) {
    return (k >> 6) * kChunkH + (((r >> 3) * 8 + ((k & 63) >> 3)) * 128) + (r & 7) * 16 + (k & 7) * 2;
}

// acc (TMEM, this warp's 32 rows, 256 columns from col0) + bias, ReLU, bf16 -> the A operand in shared memory
__device__ __forceinline__ void epilogue_hidden(uint32_t tmem_row, const float* bias, uint8_t* sH, uint32_t r) {
    for (uint32_t j0 = 0; j0 < kHidN; j0 += 16) {
        uint32_t v[16];
        tmem_ld16(tmem_row + j0, v);
        uint32_t w[8];
#pragma unroll
        for (uint32_t j = 0; j < 8; ++j) {
            const float a = fmaxf(__uint_as_float(v[2 * j]) + bias[j0 + 2 * j], 0.0f);
            const float b = fmaxf(__uint_as_float(v[2 * j + 1]) + bias[j0 + 2 * j + 1], 0.0f);
            w[j] = pack_bf16(a, b);
        }
        *reinterpret_cast<uint4*>(sH + a_off(r, j0)) = make_uint4(w[0], w[1], w[2], w[3]);
        *reinterpret_cast<uint4*>(sH + a_off(r, j0 + 8)) = make_uint4(w[4], w[5], w[6], w[7]);
    }
}

__global__ void __launch_bounds__(kInferThreads, 1) mlp_infer_kernel(InferArgs G) {
    extern __shared__ __align__(1024) uint8_t smem[];
    // barriers: 0 weights (W1, W3), 1..2 ring slot full, 3..4 ring slot free, 5 MMA done
    __shared__ __align__(8) uint64_t bars[6];
    __shared__ uint32_t tmem_base;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    const uint32_t sbase = smem_u32(smem);
    const uint32_t b_w = smem_u32(&bars[0]), b_mma = smem_u32(&bars[5]);
    auto b_full = [&](uint32_t s) { return smem_u32(&bars[1 + s]); };
    auto b_free = [&](uint32_t s) { return smem_u32(&bars[3 + s]); };
    float* sb1 = reinterpret_cast<float*>(smem + kOffBias);
    float* sb2 = sb1 + kHidN;
    float* sb3 = sb2 + kHidN;
    for (uint32_t i = tid; i < kHidN; i += kInferThreads) {
        sb1[i] = G.b1[i];
        sb2[i] = G.b2[i];
    }
    if (tid < kOutN) sb3[tid] = G.b3[tid];
    if (tid == 0) {
        for (uint32_t i = 0; i < 6; ++i) mbar_init(smem_u32(&bars[i]), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                     "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base;
    if (tid == 0) {
        // resident weights, and W2 chunks 0 and 1 into the ring
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(b_w),
                     "r"(kHidN * kInN * 2 + 4 * kChunkW3)
                     : "memory");
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                         sbase + kOffW1),
                     "l"(G.W1t), "r"(kHidN * kInN * 2), "r"(b_w)
                     : "memory");
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                         sbase + kOffW3),
                     "l"(G.W3t), "r"(4 * kChunkW3), "r"(b_w)
                     : "memory");
        expect_bytes(b_full(0), kChunkW2);
        bulk_g2s(sbase + kOffRing, G.W2t, kChunkW2, b_full(0));
        expect_bytes(b_full(1), kChunkW2);
        bulk_g2s(sbase + kOffRing + kChunkW2, reinterpret_cast<const uint8_t*>(G.W2t) + kChunkW2, kChunkW2, b_full(1));
    }
    const uint32_t idesc256 = (1u << 4) | (1u << 7) | (1u << 10) | ((kHidN >> 3) << 17) | ((128u >> 4) << 24);
    const uint32_t idesc32 = (1u << 4) | (1u << 7) | (1u << 10) | ((kOutN >> 3) << 17) | ((128u >> 4) << 24);
    uint32_t ph_mma = 0, ph_full[2] = {0, 0}, ph_free[2] = {0, 0};
    bool pending[2] = {true, true};  // (thread 0) a bulk copy into the ring slot has not been waited for
    // every exit decision is taken by the whole block (__syncthreads_and), so that
    // no thread leaves a loop that the others stay in
    bool ok = __syncthreads_and(mbar_wait(b_w, 0));
    const uint32_t n_tiles = (G.count + 127) / 128;
    uint8_t* sH = smem + kOffH;
    const uint32_t tmem_row = tmem + ((warp * 32u) << 16);
    for (uint32_t t = blockIdx.x; t < n_tiles && ok; t += gridDim.x) {
        const uint32_t r = warp * 32u + lane, row = t * 128u + r;
        // ---- X: the row's 32 features as bf16, K padded to 64 with zeros (chunk 0 of sH)
        {
            float f[32];
            if (row < G.count) {
                const float4* src = reinterpret_cast<const float4*>(G.feat + (size_t)row * 32);
#pragma unroll
                for (uint32_t q = 0; q < 8; ++q) {
                    const float4 x = src[q];
                    f[4 * q] = x.x; f[4 * q + 1] = x.y; f[4 * q + 2] = x.z; f[4 * q + 3] = x.w;
                }
            } else {
#pragma unroll
                for (uint32_t q = 0; q < 32; ++q) f[q] = 0.0f;
            }
#pragma unroll
            for (uint32_t c = 0; c < 4; ++c)
                *reinterpret_cast<uint4*>(sH + a_off(r, 8 * c)) =
                    make_uint4(pack_bf16(f[8 * c], f[8 * c + 1]), pack_bf16(f[8 * c + 2], f[8 * c + 3]),
                               pack_bf16(f[8 * c + 4], f[8 * c + 5]), pack_bf16(f[8 * c + 6], f[8 * c + 7]));
#pragma unroll
            for (uint32_t c = 4; c < 8; ++c) *reinterpret_cast<uint4*>(sH + a_off(r, 8 * c)) = make_uint4(0, 0, 0, 0);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        // ---- layer 1
        if (tid == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (uint32_t s = 0; s < 4; ++s)
                mma_bf16(tmem, smem_desc(sbase + kOffH + s * 256u), smem_desc(sbase + kOffW1 + s * 256u), idesc256,
                         s > 0);
            mma_commit(b_mma);
        }
        bool w = mbar_wait(b_mma, ph_mma);
        ph_mma ^= 1u;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (w) epilogue_hidden(tmem_row, sb1, sH, r);
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        if (!(ok = __syncthreads_and(w))) break;
        // ---- layer 2: K-chunk q of H1 against W2 chunk q from ring slot q % 2; each
        // slot refills (chunk q + 2, or chunk q - 2 for the next tile) once its MMAs end
        w = true;
        if (tid == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (uint32_t q = 0; q < 4 && w; ++q) {
                const uint32_t sl = q & 1u;
                w = mbar_wait(b_full(sl), ph_full[sl]);
                ph_full[sl] ^= 1u;
                pending[sl] = false;
                if (!w) break;
                const uint32_t slot = sbase + kOffRing + sl * kChunkW2;
#pragma unroll
                for (uint32_t s = 0; s < 4; ++s)
                    mma_bf16(tmem + kHidN, smem_desc(sbase + kOffH + q * kChunkH + s * 256u), smem_desc(slot + s * 256u),
                             idesc256, (q > 0 || s > 0) ? 1u : 0u);
                mma_commit(b_free(sl));
                if (q == 3) mma_commit(b_mma);
                if (q >= 1) {
                    const uint32_t ps = (q - 1) & 1u, nq = (q + 1) & 3u;
                    w = mbar_wait(b_free(ps), ph_free[ps]);
                    ph_free[ps] ^= 1u;
                    if (w) {
                        expect_bytes(b_full(ps), kChunkW2);
                        bulk_g2s(sbase + kOffRing + ps * kChunkW2, reinterpret_cast<const uint8_t*>(G.W2t) + nq * kChunkW2,
                                 kChunkW2, b_full(ps));
                        pending[ps] = true;
                    }
                }
            }
            if (w) {  // the slot of chunk 3 refills with chunk 1 of the next tile
                w = mbar_wait(b_free(1), ph_free[1]);
                ph_free[1] ^= 1u;
                if (w) {
                    expect_bytes(b_full(1), kChunkW2);
                    bulk_g2s(sbase + kOffRing + kChunkW2, reinterpret_cast<const uint8_t*>(G.W2t) + kChunkW2, kChunkW2,
                             b_full(1));
                    pending[1] = true;
                }
            }
        }
        if (!(ok = __syncthreads_and(w))) break;
        w = mbar_wait(b_mma, ph_mma);
        ph_mma ^= 1u;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (w) epilogue_hidden(tmem_row + kHidN, sb2, sH, r);
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        if (!(ok = __syncthreads_and(w))) break;
        // ---- layer 3
        if (tid == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (uint32_t q = 0; q < 4; ++q)
#pragma unroll
                for (uint32_t s = 0; s < 4; ++s)
                    mma_bf16(tmem, smem_desc(sbase + kOffH + q * kChunkH + s * 256u),
                             smem_desc(sbase + kOffW3 + q * kChunkW3 + s * 256u), idesc32, (q > 0 || s > 0) ? 1u : 0u);
            mma_commit(b_mma);
        }
        w = mbar_wait(b_mma, ph_mma);
        ph_mma ^= 1u;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (w) {
            uint32_t v[32];
            tmem_ld16(tmem_row, v);
            tmem_ld16(tmem_row + 16, v + 16);
            float z[32];
#pragma unroll
            for (uint32_t j = 0; j < 32; ++j) z[j] = __uint_as_float(v[j]) + sb3[j];
            if (row < G.count) {
                if (G.logits) {
                    float4* dst = reinterpret_cast<float4*>(G.logits + (size_t)row * 32);
#pragma unroll
                    for (uint32_t q = 0; q < 8; ++q) dst[q] = make_float4(z[4 * q], z[4 * q + 1], z[4 * q + 2], z[4 * q + 3]);
                }
                if (G.sel) {  // ties: the lower index
                    uint32_t bm = 0, bt = 0;
                    float zm = z[0], zt = z[kSelModes];
#pragma unroll
                    for (uint32_t k = 1; k < kSelModes; ++k)
                        if (z[k] > zm) { zm = z[k]; bm = k; }
#pragma unroll
                    for (uint32_t k = 1; k < kSelTables; ++k)
                        if (z[kSelModes + k] > zt) { zt = z[kSelModes + k]; bt = k; }
                    G.sel[row] = (uint8_t)(bm | (bt << 4));
                }
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        ok = __syncthreads_and(w);  // sH is rewritten by the next tile
    }
    if (!ok && tid == 0 && G.err) atomicExch(G.err, 1u);
    // ring copies still in flight land before the CTA exits (bounded waits)
    if (tid == 0)
        for (uint32_t sl = 0; sl < 2; ++sl)
            if (pending[sl]) mbar_wait(b_full(sl), ph_full[sl]);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
}

// A kernel's dynamic shared memory beyond 48 KB holds for the device that it was allowed on: once
// for each, noted in the kernel's `allowed`.
using AllowedOn = std::atomic<bool>[64];
template <class Kernel>
cudaError_t allow_smem(Kernel kernel, int bytes, AllowedOn& allowed) {
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess || (device < 64 && allowed[device])) return e;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess && device < 64) allowed[device] = true;
    return e;
}

}  // namespace

cudaError_t launch_mlp_infer(const float* feat, uint32_t count, const __nv_bfloat16* W1t, const __nv_bfloat16* W2t,
                             const __nv_bfloat16* W3t, const float* b1, const float* b2, const float* b3, float* logits,
                             uint8_t* sel, uint32_t* err, int device, cudaStream_t st) {
    if (count == 0) return cudaSuccess;
    static AllowedOn allowed;
    const cudaError_t e = allow_smem(mlp_infer_kernel, (int)kInferSmem, allowed);
    if (e != cudaSuccess) return e;
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    InferArgs G;
    G.feat = feat;
    G.count = count;
    G.W1t = W1t;
    G.W2t = W2t;
    G.W3t = W3t;
    G.b1 = b1;
    G.b2 = b2;
    G.b3 = b3;
    G.logits = logits;
    G.sel = sel;
    G.err = err;
    const uint32_t tiles = (count + 127) / 128;
    const uint32_t grid = std::min<uint32_t>(tiles, (uint32_t)std::max(sms, 1));
    mlp_infer_kernel<<<grid, kInferThreads, kInferSmem, st>>>(G);
    return cudaGetLastError();
}

static uint32_t gemm_blocks(const GemmArgs& g) { return g.M / 128 * ((g.N + g.tile_n - 1) / g.tile_n); }

cudaError_t launch_gemm_bf16(const GemmArgs& g, cudaStream_t st, const GemmArgs* second) {
    if (g.M == 0 || g.N == 0 || g.K == 0) return cudaSuccess;
    for (const GemmArgs* p : {&g, second})
        if (p && (p->M % 128 || p->N % 16 || p->K % kKChunk || p->tile_n == 0 || p->tile_n % 16 ||
                  p->tile_n > (p->tiled ? kTileN : kTileWide)))
            return cudaErrorInvalidValue;
    if (second && (second->tiled != g.tiled || g.tile_n > kTileN || second->tile_n > kTileN))
        return cudaErrorInvalidValue;
    constexpr int smem = (int)((kTileA + kTileB) * kStages);
    const int form = g.tiled ? 0 : (g.tile_n <= kTileN ? 1 : 2);
    const auto kernel = form == 0 ? gemm_bf16_kernel<true, false>
                                  : (form == 1 ? gemm_bf16_kernel<false, false> : gemm_bf16_kernel<false, true>);
    static AllowedOn allowed[3];
    const cudaError_t e = allow_smem(kernel, smem, allowed[form]);
    if (e != cudaSuccess) return e;
    const uint32_t n = gemm_blocks(g);
    kernel<<<n + (second ? gemm_blocks(*second) : 0u), kGemmThreads, smem, st>>>(g, second ? *second : g, n);
    return cudaGetLastError();
}

}  // namespace csv

// ---------------------------------------------------------------- C ABI
#include "abi_internal.h"

extern "C" int csv_gemm_bf16(csv_ctx* ctx, const void* d_A, const void* d_B, uint32_t M, uint32_t N, uint32_t K,
                             const float* d_bias, const void* d_mask, uint32_t relu, float* d_C, void* d_Cb,
                             void* d_CbT, float* d_CT, uint32_t* d_err, void* stream) {
    using namespace csv;
    if (!ctx || !d_A || !d_B) return CSV_EINVAL;
    if (M % 128 || N % 16 || K % 64) return abi_fail(ctx, CSV_EINVAL, "gemm: M % 128, N % 16 and K % 64 must be 0");
    DeviceGuard g(ctx->device);
    GemmArgs G;
    G.A = (const __nv_bfloat16*)d_A;
    G.B = (const __nv_bfloat16*)d_B;
    G.M = M;
    G.N = N;
    G.K = K;
    G.bias = d_bias;
    G.mask = (const __nv_bfloat16*)d_mask;
    G.relu = relu;
    G.C = d_C;
    G.Cb = (__nv_bfloat16*)d_Cb;
    G.CbT = (__nv_bfloat16*)d_CbT;
    G.CT = d_CT;
    G.err = d_err;
    // An output over an operand (a layer in place): its rows are written by the CTA that has read them, so one CTA
    // takes the row of tiles, 256 columns, as long as that is all of them.  (89,600 rows x 256 x 256: 0.134 ms, 0.119
    // beside the operands; 2048 rows 40 and 22 us.)
    auto over = [](const void* out, size_t out_bytes, const void* in, size_t in_bytes) {
        const uintptr_t a = reinterpret_cast<uintptr_t>(out), b = reinterpret_cast<uintptr_t>(in);
        return out && a < b + in_bytes && b < a + out_bytes;
    };
    auto over_operand = [&](const void* out, size_t out_bytes) {
        return over(out, out_bytes, d_A, 2 * (size_t)M * K) || over(out, out_bytes, d_B, 2 * (size_t)N * K);
    };
    const size_t mn = (size_t)M * N;
    if (over_operand(d_C, 4 * mn) || over_operand(d_CT, 4 * mn) || over_operand(d_Cb, 2 * mn) ||
        over_operand(d_CbT, 2 * mn))
        G.tile_n = kTileWide;
    cudaError_t e = launch_gemm_bf16(G, (cudaStream_t)stream);
    if (e != cudaSuccess) return abi_cuda_fail(ctx, e, "gemm");
    return CSV_OK;
}
