// selector.cu -- per-brick encoding mode and shared rANS table: the exhaustive
// search, the cheap brick statistics, and the learned selector (a 3-layer MLP
// trained and run with the tensor-core dense layer of mlp.cu).
//
// No reference counterpart: the reference encodes every brick with one op
// preference order (brickEncoding.hpp:198-282) and one rANS model per dataset
// (brickEncoding.hpp:481-482).  A version-2 image (encode.cu) names a mode and
// one of up to 16 shared tables per brick; the decoder replays any mode
// unchanged and picks the brick's table, so decode stays exact.
//
//   features_kernel    32 statistics per brick from the volume
//   select_kernel      exhaustive choice: per brick, the (mode, table) with the
//                      fewest estimated bits from the per-mode nibble histograms
//   MLP                features -> 256 -> 256 -> 12 mode logits + 16 table logits;
//                      bf16 weights, fp32 accumulation (tcgen05), Adam in fp32
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <new>
#include <string>
#include <vector>

#include "abi_internal.h"
#include "csv_internal.h"
#include "majority.cuh"

namespace csv {
namespace {

constexpr uint32_t kFeat = 32, kFeatPad = 64, kHid = 256, kOut = 32, kOutPad = 64;
constexpr uint32_t kModesN = 12, kTablesN = 16;
constexpr uint32_t kFThreads = 256;

__device__ __forceinline__ uint32_t spread3(uint32_t v) {
    v &= 0x3ffu;
    v = (v | (v << 16)) & 0x030000ffu;
    v = (v | (v << 8)) & 0x0300f00fu;
    v = (v | (v << 4)) & 0x030c30c3u;
    v = (v | (v << 2)) & 0x09249249u;
    return v;
}

struct FeatShared {
    uint64_t lab[585];       // the 8^3 sample's pyramid: levels 0 .. 3 (the sample, Morton order)
    uint32_t slot[1024];     // hash table of the sample: 1 + the index of a label's first holder
    uint8_t cst[73];         // constant flags of levels 0 .. 2
    uint32_t cnt[16];        // eq1 x y z, eq4 x y z, zeros, runs per bucket [7], runs
    uint32_t distinct;
};

__device__ __forceinline__ uint64_t vox(const uint64_t* vol, uint64_t W, uint64_t H, uint64_t D, uint64_t x, uint64_t y,
                                        uint64_t z) {
    return (x < W && y < H && z < D) ? __ldg(vol + x + W * (y + H * z)) : 0ull;  // padding, brick.hpp:181-183
}

__device__ __forceinline__ uint32_t bitlen(uint32_t v) { return v ? 32u - __clz(v) : 0u; }

// Mini-brick op histogram: encodeBrick's op choice (mode 0, brickEncoding.hpp:188-447)
// on the 8^3 sample, by one warp, 32 children at a time in stream order.  Nibbles
// counted: root, every op, Pd offsets; lane v returns the count of nibble v.  The palette
// ops of a group are settled as the encoder's palette walk does: all lanes look their
// label up in the window of the last 17 entries, then one step per miss.
__device__ uint32_t mini_ops(const FeatShared& S) {
    const uint32_t FULL = 0xFFFFFFFFu, lane = threadIdx.x & 31u;
    const bool root_const = S.cst[0] != 0;
    uint32_t count = lane == ((4u << 1) | (root_const ? 1u : 0u)) ? 1u : 0u;
    if (root_const) return count;
    auto at = [&](uint32_t l, uint32_t m) -> uint64_t { return S.lab[((1u << (3 * l)) - 1) / 7 + m]; };
    uint64_t win = lane == 0 ? S.lab[0] : 0;
    uint32_t P = 1;
    for (uint32_t k0 = 1; k0 < 585; k0 += 32) {  // nodes of levels 1 .. 3, in order
        const uint32_t k = k0 + lane;
        uint32_t code = 8, stop = 0;  // 8: no op here
        uint64_t mine = 0;
        if (k < 585) {
            const uint32_t lc = k < 9 ? 1u : (k < 73 ? 2u : 3u), l = lc - 1;
            const uint32_t n = k - ((1u << (3 * lc)) - 1) / 7, p = n >> 3, lvlmask = (1u << (3 * lc)) - 1u;
            if (!S.cst[((1u << (3 * l)) - 1) / 7 + p]) {
                mine = S.lab[k];
                stop = lc == 3 ? 1u : S.cst[k];
                code = at(l, p) == mine ? 0u : 7u;
#pragma unroll
                for (uint32_t a = 0; a < 3; ++a) {
                    const uint32_t m = (0x09249249u << a) & lvlmask, bit = 1u << a;
                    if (n & bit) {
                        if ((n & m) == m) continue;
                        const uint32_t N = (((n | ~m) + bit) & m) | (n & ~m);
                        if (code == 7 && at(l, N >> 3) == mine) code = 1 + a;
                    } else {
                        if ((n & m) == 0) continue;
                        const uint32_t N = (((n & m) - bit) & m) | (n & ~m);
                        if (code == 7 && at(lc, N) == mine) code = 1 + a;
                    }
                }
            }
        }
        uint32_t delta = 16;  // of a Pd op
        const bool need = code == 7;
        if (__ballot_sync(FULL, need)) {
            int d = -1;
            const uint32_t depth = min(P, 17u);
            for (uint32_t e = 0; e < depth; ++e)
                if (__shfl_sync(FULL, win, e) == mine) d = (int)e;
            bool added = false;
            for (uint32_t miss = __ballot_sync(FULL, need && d < 0); miss;) {
                const uint32_t f = __ffs(miss) - 1;
                const uint64_t entry = __shfl_sync(FULL, mine, f), up = __shfl_up_sync(FULL, win, 1);
                win = lane == 0 ? entry : up;
                ++P;
                if (lane == f) added = true;
                if (lane > f) d = mine == entry ? 0 : (d >= 0 && d < 16 ? d + 1 : -1);
                miss = __ballot_sync(FULL, need && lane > f && d < 0);
            }
            if (need) {
                code = added ? 4u : (d == 0 ? 5u : 6u);
                if (code == 6) delta = (uint32_t)d - 1;
            }
        }
        auto add = [&](uint32_t v, bool has) {  // lane b counts the lanes with v == b
            uint32_t m = __ballot_sync(FULL, has);
#pragma unroll
            for (uint32_t q = 0; q < 4; ++q) {
                const uint32_t bb = __ballot_sync(FULL, (v >> q) & 1u);
                m &= (lane >> q) & 1u ? bb : ~bb;
            }
            if (lane < 16) count += __popc(m);
        };
        add(code << 1 | stop, code < 8);
        if (__ballot_sync(FULL, delta < 16)) add(delta, delta < 16);
    }
    return count;
}

// The statistics of the 8^3 sample at the centres of the brick's 8^3 cells: distinct
// labels (S.distinct) and, in the first warp, the op nibbles.
__device__ uint32_t sample_stats(FeatShared& S, const uint64_t* vol, uint64_t W, uint64_t H, uint64_t D, uint64_t x0,
                                 uint64_t y0, uint64_t z0, uint32_t b) {
    const uint32_t tid = threadIdx.x;
    const uint32_t step = b / 8, off = step / 2;
    for (uint32_t k = tid; k < 1024; k += kFThreads) S.slot[k] = 0;
    for (uint32_t k = tid; k < 512; k += kFThreads) {
        const uint32_t x = k & 7u, y = (k >> 3) & 7u, z = k >> 6;
        const uint32_t m = spread3(x) | (spread3(y) << 1) | (spread3(z) << 2);
        S.lab[73 + m] = vox(vol, W, H, D, x0 + x * step + off, y0 + y * step + off, z0 + z * step + off);
    }
    if (tid == 0) S.distinct = 0;
    __syncthreads();
    uint32_t fresh = 0;
    for (uint32_t k = tid; k < 512; k += kFThreads) {  // linear probing; at least half the slots stay free
        const uint64_t v = S.lab[73 + k];
        uint32_t h = (((uint32_t)v * 0x9E3779B1u) ^ ((uint32_t)(v >> 32) * 0x85EBCA77u)) >> 22;
        for (uint32_t tries = 0; tries < 1024; ++tries) {
            const uint32_t was = atomicCAS(&S.slot[h], 0u, k + 1);
            if (was == 0) {
                ++fresh;
                break;
            }
            if (S.lab[73 + was - 1] == v) break;
            h = (h + 1) & 1023u;
        }
    }
    if (fresh) atomicAdd(&S.distinct, fresh);
    // the pyramid (Brick::build on 8^3): levels 2, 1, 0, by the first two warps
    for (int l = 2; l >= 0; --l) {
        const uint32_t cntl = 1u << (3 * l), here = ((1u << (3 * l)) - 1) / 7, below = ((8u << (3 * l)) - 1) / 7;
        if (tid < cntl) {
            uint64_t v[8];
            bool same, cc = true;
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = S.lab[below + 8 * tid + k];
            if (l < 2)
                for (int k = 0; k < 8; ++k) cc &= S.cst[below + 8 * tid + k] != 0;
            S.lab[here + tid] = majority8(v, same);
            S.cst[here + tid] = same && cc ? 1 : 0;
        }
        __syncthreads();
    }
    return tid < 32 ? mini_ops(S) : 0u;
}

// Statistics of the bricks, `parts` CTAs per brick (few bricks: more, so that every SM
// has rows to read).  A CTA counts over its part of the rows of even y and even z (all x:
// a quarter of the voxels, every pair within such a row, and each such voxel's +1 / +4
// neighbours in y and z), a row per warp at a time with its four neighbour rows read
// beside it, so that ten loads per lane are in flight.  The sample's statistics, a serial
// walk, are a CTA of their own, and these come first (one CTA does both where a brick has
// one).  Counts meet in the brick's feature row as whole numbers (zeroed by the launch);
// the last CTA to add its own turns them into the features.
// Row words: 0 .. 14 counts, 15 CTAs done | distinct << 16, 16 .. 31 op nibbles.
// Measured (B200, 320 bricks of 64^3): 0.41 -> 0.156 ms (one CTA per brick with planes
// kept in registers, the runs counted start by start and the sample's ops walked by one
// thread; 0.170 ms, and 66 for 47 us with 64 bricks, with the sample in a CTA that has rows
// too); the rows it reads are three quarters of the volume, 0.08 ms at the HBM rate.
__global__ void __launch_bounds__(kFThreads, 4) features_kernel(const uint64_t* __restrict__ vol, uint64_t W, uint64_t H,
                                                                uint64_t D, uint32_t b, uint32_t nbx, uint32_t nby,
                                                                uint32_t nbz, uint32_t parts, float* __restrict__ feat) {
    __shared__ FeatShared S;
    const uint32_t nb = nbx * nby * nbz, shares = parts > 1 ? parts - 1 : 1;
    const bool sample = parts == 1 || blockIdx.x < nb, rows = parts == 1 || !sample;
    const uint32_t j = parts == 1 || sample ? blockIdx.x : blockIdx.x - nb;
    const uint32_t i = parts == 1 || sample ? j : j / shares, part = parts == 1 || sample ? 0 : j % shares;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t bz = i % nbz, by = (i / nbz) % nby, bx = i / (nbz * nby);  // split order (brick.hpp:152-154)
    const uint64_t x0 = (uint64_t)bx * b, y0 = (uint64_t)by * b, z0 = (uint64_t)bz * b;
    uint32_t* row_out = reinterpret_cast<uint32_t*>(feat + (size_t)i * kFeat);
    if (tid < 16) S.cnt[tid] = 0;
    uint32_t nibbles = 0;
    if (sample) nibbles = sample_stats(S, vol, W, H, D, x0, y0, z0, b);
    __syncthreads();
    uint32_t c[15] = {};
    // a row's runs follow from the mask of their starts: lane l keeps the mask of the warp's row l, and
    // every 32 rows the lanes take theirs apart
    uint64_t row_starts = 0;
    uint32_t rows_kept = 0;
    auto count_runs = [&]() {
        const uint64_t s = row_starts;
        if (lane < rows_kept) {
            const uint32_t n = __popcll(s);
            c[14] += n;
            c[0] += b - n;  // a voxel that starts no run equals its left neighbour
            // cumulative: runs with another start, or the row's end, within 1, 2, 4, .. voxels of theirs
            uint64_t near = (s >> 1) | (1ull << (b - 1));
            uint32_t below = 0;
#pragma unroll
            for (uint32_t k = 0; k < 6; ++k) {
                const uint32_t m = __popcll(s & near);
                c[7 + k] += m - below;
                below = m;
                near |= near >> (1u << k);
            }
            c[13] += n - below;
        }
        rows_kept = 0;
    };
    if (rows) {
        const uint32_t nch = (b + 31) / 32;  // values per lane: 1 or 2 (lane l holds x = l and x = l + 32)
        const bool interior = x0 + b <= W && y0 + b <= H && z0 + b <= D;
        const uint64_t WH = W * H;
        const uint32_t hb = b / 2, items = hb * hb, per = (items + shares - 1) / shares;
        const uint32_t it1 = min(items, (part + 1) * per);
        for (uint32_t it = part * per + warp; it < it1; it += kFThreads / 32) {
            const uint32_t y = 2 * (it % hb), z = 2 * (it / hb);
            const bool far_y = y + 4 < b, far_z = z + 4 < b;
            uint64_t v[2], y1[2], z1[2], y4[2], z4[2];
            const uint64_t* p = vol + (x0 + lane + W * (y0 + y) + WH * (z0 + z));
#pragma unroll
            for (uint32_t h = 0; h < 2; ++h) {
                const uint32_t x = lane + 32 * h;
                v[h] = y1[h] = z1[h] = y4[h] = z4[h] = 0ull;
                if (h < nch && x < b) {
                    if (interior) {
                        const uint64_t* q = p + 32 * h;
                        v[h] = __ldg(q);
                        y1[h] = __ldg(q + W);
                        z1[h] = __ldg(q + WH);
                        if (far_y) y4[h] = __ldg(q + 4 * W);
                        if (far_z) z4[h] = __ldg(q + 4 * WH);
                    } else {
                        const uint64_t gx = x0 + x, gy = y0 + y, gz = z0 + z;
                        v[h] = vox(vol, W, H, D, gx, gy, gz);
                        y1[h] = vox(vol, W, H, D, gx, gy + 1, gz);
                        z1[h] = vox(vol, W, H, D, gx, gy, gz + 1);
                        y4[h] = vox(vol, W, H, D, gx, gy + 4, gz);
                        z4[h] = vox(vol, W, H, D, gx, gy, gz + 4);
                    }
                }
            }
            // x + 4 and x - 1 from the lanes that hold them
            const uint64_t up0 = __shfl_up_sync(0xffffffffu, v[0], 1), up1 = __shfl_up_sync(0xffffffffu, v[1], 1),
                           wrap1 = __shfl_sync(0xffffffffu, v[0], 31);
            const uint64_t d0 = __shfl_down_sync(0xffffffffu, v[0], 4), d1 = __shfl_down_sync(0xffffffffu, v[1], 4),
                           wrap4 = __shfl_sync(0xffffffffu, v[1], (lane + 4) & 31u);
            uint64_t starts = 0;
#pragma unroll
            for (uint32_t h = 0; h < 2; ++h) {
                const uint32_t x = lane + 32 * h;
                const bool in = h < nch && x < b;
                const uint64_t x4 = h ? d1 : (lane < 28 ? d0 : wrap4), left = h ? (lane ? up1 : wrap1) : up0;
                if (in) {
                    c[1] += v[h] == y1[h];
                    c[2] += v[h] == z1[h];
                    c[3] += x + 4 < b && v[h] == x4;
                    c[4] += far_y && v[h] == y4[h];
                    c[5] += far_z && v[h] == z4[h];
                    c[6] += v[h] == 0;
                }
                starts |= (uint64_t)__ballot_sync(0xffffffffu, in && (x == 0 || left != v[h])) << (32 * h);
            }
            if (lane == rows_kept) row_starts = starts;
            if (++rows_kept == 32) count_runs();
        }
    }
    count_runs();
#pragma unroll
    for (int k = 0; k < 15; ++k) {
        const uint32_t v = __reduce_add_sync(0xffffffffu, c[k]);
        if (lane == 0 && v) atomicAdd(&S.cnt[k], v);
    }
    __syncthreads();
    if (warp == 0) {
        if (sample && lane < 16) atomicExch(row_out + 16 + lane, nibbles);
        if (lane < 15 && S.cnt[lane]) atomicAdd(row_out + lane, S.cnt[lane]);
        __threadfence();
        __syncwarp();
        uint32_t done = 0;
        if (lane == 0) done = atomicAdd(row_out + 15, 1u + (sample ? S.distinct << 16 : 0u));
        done = __shfl_sync(0xffffffffu, done, 0);
        if ((done & 0xFFFFu) + 1 != parts) return;
        __threadfence();
        const uint32_t mine = __ldcg(row_out + lane);
        const uint32_t w15 = __shfl_sync(0xffffffffu, mine, 15), n_runs = __shfl_sync(0xffffffffu, mine, 14);
        const uint32_t tot = __reduce_add_sync(0xffffffffu, lane >= 16 ? mine : 0u);
        const uint32_t before = __shfl_up_sync(0xffffffffu, mine, 1);  // feature k holds count k - 1
        // pairs tested: x within the sampled rows; y and z from the sampled rows outward
        const float hb = (float)(b / 2), fb = (float)b;
        const float px1 = hb * hb * (fb - 1.0f), px4 = hb * hb * (fb - 4.0f);
        const float pyz1 = hb * hb * fb, pyz4 = (float)((b - 4) / 2) * hb * fb;
        float f;
        if (lane == 0) f = (float)bitlen(w15 >> 16) / 10.0f;
        else if (lane == 1) f = (float)before / px1;
        else if (lane <= 3) f = (float)before / pyz1;
        else if (lane == 4) f = (float)before / px4;
        else if (lane <= 6) f = (float)before / pyz4;
        else if (lane == 7) f = (float)before / (hb * hb * fb);
        else if (lane <= 14) f = (float)before / (float)max(n_runs, 1u);
        else if (lane == 15) f = (float)bitlen(n_runs) / 20.0f;
        else f = (float)mine / (float)max(tot, 1u);
        __syncwarp();
        reinterpret_cast<float*>(row_out)[lane] = f;
    }
}

// Exhaustive choice: the (mode, table) with the fewest estimated bits,
// sum_s hist[mode][s] * len[table][s] (len: bits per symbol, 16.16 fixed point);
// ties go to the lower mode, then the lower table.
// A warp per brick, its (mode, table) pairs over the lanes (150 bricks 41 -> 7 us against
// a thread per brick).
constexpr uint32_t kSelWarps = 4;
struct CodeLengths {
    uint32_t v[kTablesN * 16];
};
__global__ void __launch_bounds__(32 * kSelWarps) select_kernel(const uint32_t* __restrict__ hist, uint32_t nb,
                                                                 const CodeLengths lens, uint32_t n_tables,
                                                                 uint8_t* __restrict__ sel,
                                                                 uint64_t* __restrict__ cost_out) {
    __shared__ uint32_t len[kTablesN][17], h[kSelWarps][kModesN * 16];
    for (uint32_t k = threadIdx.x; k < kTablesN * 16; k += 32 * kSelWarps) len[k >> 4][k & 15u] = lens.v[k];
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5, i = blockIdx.x * kSelWarps + w;
    if (i < nb)
        for (uint32_t k = lane; k < kModesN * 16; k += 32) h[w][k] = hist[(size_t)i * kModesN * 16 + k];
    __syncthreads();
    if (i >= nb) return;
    uint64_t best = ~0ull;
    uint32_t pair = ~0u;  // mode * n_tables + table: the order of ties
    for (uint32_t k = lane; k < kModesN * n_tables; k += 32) {
        const uint32_t m = k / n_tables, t = k % n_tables;
        uint64_t c = 0;
#pragma unroll
        for (uint32_t s = 0; s < 16; ++s) c += (uint64_t)h[w][16 * m + s] * len[t][s];
        if (cost_out) cost_out[(size_t)i * kModesN * n_tables + k] = c;
        if (c < best) {
            best = c;
            pair = k;
        }
    }
    for (int d = 16; d > 0; d >>= 1) {
        const uint64_t c = __shfl_xor_sync(0xFFFFFFFFu, best, d);
        const uint32_t k = __shfl_xor_sync(0xFFFFFFFFu, pair, d);
        if (c < best || (c == best && k < pair)) {
            best = c;
            pair = k;
        }
    }
    if (lane == 0) sel[i] = (uint8_t)(pair / n_tables | (pair % n_tables) << 4);
}

// ---------------------------------------------------------------- MLP kernels
// Parameters, fp32, one array: W1 [256][64] (input columns 32..63 stay 0), b1 [256],
// W2 [256][256], b2 [256], W3 [32][256] (rows 28..31 stay 0), b3 [32].
constexpr uint32_t OFF_W1 = 0, OFF_B1 = OFF_W1 + kHid * kFeatPad, OFF_W2 = OFF_B1 + kHid,
                   OFF_B2 = OFF_W2 + kHid * kHid, OFF_W3 = OFF_B2 + kHid, OFF_B3 = OFF_W3 + kOut * kHid,
                   N_PARAMS = OFF_B3 + kOut;
static_assert(N_PARAMS == CSV_MLP_PARAMS, "parameter layout");

// features (n x 32, fp32) -> X (rows x 64, bf16, zero padded) and X^T (64 x rows), tiled
__global__ void pack_input_kernel(const float* __restrict__ feat, uint32_t n, uint32_t rows,
                                  __nv_bfloat16* __restrict__ X, __nv_bfloat16* __restrict__ XT) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= rows * kFeatPad) return;
    const uint32_t r = k / kFeatPad, c = k % kFeatPad;
    const float v = (r < n && c < kFeat) ? feat[(size_t)r * kFeat + c] : 0.0f;
    const __nv_bfloat16 b = __float2bfloat16_rn(v);
    X[tiled_at(rows, r, c)] = b;
    XT[tiled_at(kFeatPad, c, r)] = b;
}

// Partial sums over the rows of dZ (32 columns), dH2 and dH1 (256), the bias gradients, from
// their tiled transposes (eight rows of a column are 16 bytes): block (part, matrix), a
// thread per column, over `per` rows each (a multiple of 8, as the batch's).
__global__ void __launch_bounds__(256) colsum_kernel(const __nv_bfloat16* __restrict__ dZT,
                                                     const __nv_bfloat16* __restrict__ dH2T,
                                                     const __nv_bfloat16* __restrict__ dH1T, uint32_t rows, uint32_t per,
                                                     float* __restrict__ out) {
    const uint32_t c = threadIdx.x, which = blockIdx.y, cols = which == 0 ? kOut : kHid;
    if (c >= cols) return;
    const __nv_bfloat16* m = which == 0 ? dZT : (which == 1 ? dH2T : dH1T);
    const uint32_t r1 = min(rows, (blockIdx.x + 1) * per);
    float s = 0.0f;
#pragma unroll 4
    for (uint32_t r = blockIdx.x * per; r < r1; r += 8) {
        const uint4 v = *reinterpret_cast<const uint4*>(m + tiled_at(cols, c, r));
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {  // (bf16 is the upper half of fp32)
            s += __uint_as_float(w[k] << 16);
            s += __uint_as_float(w[k] & 0xFFFF0000u);
        }
    }
    out[((size_t)which * gridDim.x + blockIdx.x) * kHid + c] = s;
}

// The bias gradients from colsum_kernel's partial sums, in order.
__global__ void __launch_bounds__(256) bias_sum_kernel(const float* __restrict__ part, uint32_t parts,
                                                       float* __restrict__ G) {
    const uint32_t c = threadIdx.x, which = blockIdx.x;
    if (which == 0 && c >= kOut) return;
    float s = 0.0f;
#pragma unroll 8
    for (uint32_t i = 0; i < parts; ++i) s += part[((size_t)which * parts + i) * kHid + c];
    G[(which == 0 ? OFF_B3 : (which == 1 ? OFF_B2 : OFF_B1)) + c] = s;
}

// A weight's bf16 copies, tiled as the layers read them: W1 [256][64], W2 [256][256] and its
// transpose, W3 [32][256] and its transpose [256][64] (columns >= 32 zero).
struct WeightCopies {
    __nv_bfloat16 *W1t, *W2t, *W2Tt, *W3t, *W3Tt;
};
__device__ __forceinline__ void put_weight(const WeightCopies& C, uint32_t k, float v) {
    const __nv_bfloat16 w = __float2bfloat16_rn(v);
    if (k < OFF_B1) {
        C.W1t[tiled_at(kHid, k / kFeatPad, k % kFeatPad)] = w;
    } else if (k >= OFF_W2 && k < OFF_B2) {
        const uint32_t i = k - OFF_W2, o = i / kHid, in = i % kHid;
        C.W2t[tiled_at(kHid, o, in)] = w;
        C.W2Tt[tiled_at(kHid, in, o)] = w;
    } else if (k >= OFF_W3 && k < OFF_B3) {
        const uint32_t i = k - OFF_W3, o = i / kHid, in = i % kHid;
        C.W3t[tiled_at(kOut, o, in)] = w;
        C.W3Tt[tiled_at(kHid, in, o)] = w;
    }
}

// Adam (Kingma & Ba 2015) on the fp32 parameters, and the weights' bf16 copies.
__global__ void adam_kernel(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                            float* __restrict__ v, uint32_t n, float lr, float b1, float b2, float eps, float c1,
                            float c2, WeightCopies C) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const float gk = g[k];
    const float mk = b1 * m[k] + (1.0f - b1) * gk, vk = b2 * v[k] + (1.0f - b2) * gk * gk;
    m[k] = mk;
    v[k] = vk;
    const float pk = p[k] - lr * (mk / c1) / (sqrtf(vk / c2) + eps);
    p[k] = pk;
    put_weight(C, k, pk);
}

// The copies of given parameters.
__global__ void refresh_kernel(const float* __restrict__ P, WeightCopies C) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < N_PARAMS) put_weight(C, k, P[k]);
    if (k < kHid * (kOutPad - kOut)) {
        const uint32_t in = k / (kOutPad - kOut), o = kOut + k % (kOutPad - kOut);
        C.W3Tt[tiled_at(kHid, in, o)] = __float2bfloat16_rn(0.0f);
    }
}

}  // namespace
}  // namespace csv

// ---------------------------------------------------------------- network and C ABI
using namespace csv;

struct csv_mlp {
    csv_ctx* ctx = nullptr;
    uint32_t cap = 0;  // batch rows the activations hold (multiple of 128)
    uint32_t t = 0;    // Adam steps taken
    float* P = nullptr;  // parameters, gradients, Adam moments (N_PARAMS each)
    float* G = nullptr;
    float* Mm = nullptr;
    float* Vm = nullptr;
    __nv_bfloat16 *W1t = nullptr, *W2t = nullptr, *W2Tt = nullptr, *W3t = nullptr, *W3Tt = nullptr;  // WeightCopies
    // tiled operands of the gradient step, with their transposes
    __nv_bfloat16 *X = nullptr, *XT = nullptr, *H1 = nullptr, *H1T = nullptr, *H2 = nullptr, *H2T = nullptr;
    __nv_bfloat16 *dZ = nullptr, *dZT = nullptr, *dH2 = nullptr, *dH2T = nullptr, *dH1T = nullptr;
    float* bias_part = nullptr;  // the bias gradients' partial sums
    float* loss = nullptr;
    uint32_t* err = nullptr;
};

namespace {

void mlp_free_acts(csv_mlp* n) {
    for (void* p : {(void*)n->X, (void*)n->XT, (void*)n->H1, (void*)n->H1T, (void*)n->H2, (void*)n->H2T,
                    (void*)n->dZ, (void*)n->dZT, (void*)n->dH2, (void*)n->dH2T, (void*)n->dH1T,
                    (void*)n->bias_part})
        cudaFree(p);
    n->X = n->XT = n->H1 = n->H1T = n->H2 = n->H2T = n->dZ = n->dZT = n->dH2 = n->dH2T = n->dH1T = nullptr;
    n->bias_part = nullptr;
    n->cap = 0;
}

uint32_t mlp_bias_rows(uint32_t rows) { return std::max(64u, (rows / 64 + 7) / 8 * 8); }  // per partial sum
uint32_t mlp_bias_parts(uint32_t rows) { return (rows + mlp_bias_rows(rows) - 1) / mlp_bias_rows(rows); }

cudaError_t mlp_reserve(csv_mlp* n, uint32_t rows) {
    if (rows <= n->cap) return cudaSuccess;
    mlp_free_acts(n);
    const size_t r = rows;
    cudaError_t e = cudaSuccess;
    auto al = [&](void** p, size_t bytes) {
        if (e == cudaSuccess) e = cudaMalloc(p, bytes);
    };
    al((void**)&n->X, r * kFeatPad * 2);
    al((void**)&n->XT, r * kFeatPad * 2);
    al((void**)&n->H1, r * kHid * 2);
    al((void**)&n->H1T, r * kHid * 2);
    al((void**)&n->H2, r * kHid * 2);
    al((void**)&n->H2T, r * kHid * 2);
    al((void**)&n->dZ, r * kOutPad * 2);
    al((void**)&n->dZT, r * kOut * 2);
    al((void**)&n->dH2, r * kHid * 2);
    al((void**)&n->dH2T, r * kHid * 2);
    al((void**)&n->dH1T, r * kHid * 2);
    al((void**)&n->bias_part, 3 * std::min<size_t>(64, (rows + 63) / 64) * kHid * 4);
    if (e == cudaSuccess) n->cap = rows;
    return e;
}

WeightCopies mlp_copies(const csv_mlp* n) {
    return WeightCopies{n->W1t, n->W2t, n->W2Tt, n->W3t, n->W3Tt};
}

GemmArgs mlp_gemm(const csv_mlp* n, const __nv_bfloat16* A, const __nv_bfloat16* B, uint32_t M, uint32_t N, uint32_t K) {
    GemmArgs g;
    g.A = A;
    g.B = B;
    g.M = M;
    g.N = N;
    g.K = K;
    g.tiled = true;
    g.err = n->err;
    return g;
}

// Forward pass on `rows` (padded) rows of which `cnt` hold features, the loss, and dZ.
cudaError_t mlp_forward(csv_mlp* n, const float* feat, const uint8_t* label, uint32_t cnt, uint32_t rows, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(n->loss, 0, 4, st);
    if (e != cudaSuccess) return e;
    pack_input_kernel<<<(rows * kFeatPad + 255) / 256, 256, 0, st>>>(feat, cnt, rows, n->X, n->XT);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    GemmArgs g = mlp_gemm(n, n->X, n->W1t, rows, kHid, kFeatPad);
    g.bias = n->P + OFF_B1;
    g.relu = 1;
    g.Cb = n->H1;
    g.CbT = n->H1T;
    if ((e = launch_gemm_bf16(g, st)) != cudaSuccess) return e;
    g = mlp_gemm(n, n->H1, n->W2t, rows, kHid, kHid);
    g.bias = n->P + OFF_B2;
    g.relu = 1;
    g.Cb = n->H2;
    g.CbT = n->H2T;
    if ((e = launch_gemm_bf16(g, st)) != cudaSuccess) return e;
    g = mlp_gemm(n, n->H2, n->W3t, rows, kOut, kHid);
    g.bias = n->P + OFF_B3;
    g.Cb = n->dZ;
    g.CbT = n->dZT;
    g.label = label;
    g.n_rows = cnt;
    g.loss = n->loss;
    return launch_gemm_bf16(g, st);
}

}  // namespace

extern "C" {

void csv_mlp_destroy(csv_mlp* n) {
    if (!n) return;
    DeviceGuard g(n->ctx->device);
    mlp_free_acts(n);
    for (void* p : {(void*)n->P, (void*)n->G, (void*)n->Mm, (void*)n->Vm, (void*)n->W1t, (void*)n->W2t, (void*)n->W2Tt,
                    (void*)n->W3t, (void*)n->W3Tt, (void*)n->loss, (void*)n->err})
        cudaFree(p);
    delete n;
}

int csv_mlp_create(csv_ctx* ctx, const float* params, csv_mlp** out) {
    if (!ctx || !params || !out) return CSV_EINVAL;
    *out = nullptr;
    DeviceGuard g(ctx->device);
    csv_mlp* n = new (std::nothrow) csv_mlp();
    if (!n) return abi_fail(ctx, CSV_ENOMEM, "mlp: host allocation");
    n->ctx = ctx;
    cudaError_t e = cudaSuccess;
    auto al = [&](void** p, size_t bytes) {
        if (e == cudaSuccess) e = cudaMalloc(p, bytes);
    };
    al((void**)&n->P, N_PARAMS * 4);
    al((void**)&n->G, N_PARAMS * 4);
    al((void**)&n->Mm, N_PARAMS * 4);
    al((void**)&n->Vm, N_PARAMS * 4);
    al((void**)&n->W2Tt, kHid * kHid * 2);
    al((void**)&n->W3Tt, kHid * kOutPad * 2);
    al((void**)&n->W1t, kHid * kFeatPad * 2);
    al((void**)&n->W2t, kHid * kHid * 2);
    al((void**)&n->W3t, kOut * kHid * 2);
    al((void**)&n->loss, 4);
    al((void**)&n->err, 4);
    if (e == cudaSuccess) e = cudaMemcpy(n->P, params, N_PARAMS * 4, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemset(n->Mm, 0, N_PARAMS * 4);
    if (e == cudaSuccess) e = cudaMemset(n->Vm, 0, N_PARAMS * 4);
    if (e == cudaSuccess) e = cudaMemset(n->G, 0, N_PARAMS * 4);
    if (e == cudaSuccess) e = cudaMemset(n->err, 0, 4);
    if (e == cudaSuccess) {
        refresh_kernel<<<(N_PARAMS + 255) / 256, 256>>>(n->P, mlp_copies(n));
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e != cudaSuccess) {
        csv_mlp_destroy(n);
        return abi_cuda_fail(ctx, e, "mlp create");
    }
    *out = n;
    return CSV_OK;
}

int csv_mlp_params(const csv_mlp* n, float* params, float* grads) {
    if (!n) return CSV_EINVAL;
    DeviceGuard g(n->ctx->device);
    cudaError_t e = cudaDeviceSynchronize();
    if (e == cudaSuccess && params) e = cudaMemcpy(params, n->P, N_PARAMS * 4, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess && grads) e = cudaMemcpy(grads, n->G, N_PARAMS * 4, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return abi_cuda_fail(n->ctx, e, "mlp params");
    return CSV_OK;
}

int csv_mlp_forward(csv_mlp* n, const float* d_feat, uint32_t count, float* d_logits, uint8_t* d_sel, void* stream) {
    if (!n || (count && !d_feat)) return CSV_EINVAL;
    if (count == 0) return CSV_OK;
    DeviceGuard g(n->ctx->device);
    if ((reinterpret_cast<uintptr_t>(d_feat) | reinterpret_cast<uintptr_t>(d_logits)) & 15u)
        return abi_fail(n->ctx, CSV_EINVAL, "mlp forward: features and logits must be 16-byte aligned");
    cudaStream_t st = (cudaStream_t)stream;
    // the fused forward: features in, logits / choices out, activations on chip
    cudaError_t e = launch_mlp_infer(d_feat, count, n->W1t, n->W2t, n->W3t, n->P + OFF_B1, n->P + OFF_B2, n->P + OFF_B3,
                                     d_logits, d_sel, n->err, n->ctx->device, st);
    if (e != cudaSuccess) return abi_cuda_fail(n->ctx, e, "mlp forward");
    return CSV_OK;
}

int csv_mlp_grad(csv_mlp* n, const float* d_feat, const uint8_t* d_label, uint32_t count, float* loss, void* stream) {
    if (!n || !d_feat || !d_label || count == 0) return CSV_EINVAL;
    DeviceGuard g(n->ctx->device);
    cudaStream_t st = (cudaStream_t)stream;
    const uint32_t rows = (count + 127) / 128 * 128;
    cudaError_t e = mlp_reserve(n, rows);
    if (e == cudaSuccess) e = mlp_forward(n, d_feat, d_label, count, rows, st);
    // a product over the rows (few outputs, so narrow tiles) beside one over the units where both have
    // their operands
    auto over_rows = [&](const __nv_bfloat16* A, const __nv_bfloat16* B, uint32_t N) {
        GemmArgs g = mlp_gemm(n, A, B, kHid, N, rows);
        g.tile_n = 16;
        return g;
    };
    if (e == cudaSuccess) {
        GemmArgs w = over_rows(n->H2T, n->dZT, kOut);  // dW3^T = H2^T dZ, written as W3 lies
        w.CT = n->G + OFF_W3;
        GemmArgs h = mlp_gemm(n, n->dZ, n->W3Tt, rows, kHid, kOutPad);  // dH2 = (dZ W3) * (H2 > 0)
        h.mask = n->H2;
        h.Cb = n->dH2;
        h.CbT = n->dH2T;
        e = launch_gemm_bf16(w, st, &h);
    }
    if (e == cudaSuccess) {
        GemmArgs w = over_rows(n->dH2T, n->H1T, kHid);  // dW2 = dH2^T H1
        w.C = n->G + OFF_W2;
        GemmArgs h = mlp_gemm(n, n->dH2, n->W2Tt, rows, kHid, kHid);  // dH1 = (dH2 W2) * (H1 > 0)
        h.mask = n->H1;
        h.CbT = n->dH1T;
        e = launch_gemm_bf16(w, st, &h);
    }
    if (e == cudaSuccess) {
        GemmArgs w = over_rows(n->dH1T, n->XT, kFeatPad);  // dW1 = dH1^T X
        w.C = n->G + OFF_W1;
        e = launch_gemm_bf16(w, st);
    }
    if (e == cudaSuccess) {
        const uint32_t parts = mlp_bias_parts(rows);
        colsum_kernel<<<dim3(parts, 3), 256, 0, st>>>(n->dZT, n->dH2T, n->dH1T, rows, mlp_bias_rows(rows), n->bias_part);
        bias_sum_kernel<<<3, 256, 0, st>>>(n->bias_part, parts, n->G);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess && loss) {
        e = cudaMemcpyAsync(loss, n->loss, 4, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    }
    if (e != cudaSuccess) return abi_cuda_fail(n->ctx, e, "mlp grad");
    return CSV_OK;
}

int csv_mlp_adam(csv_mlp* n, float lr, float beta1, float beta2, float eps, void* stream) {
    if (!n) return CSV_EINVAL;
    DeviceGuard g(n->ctx->device);
    cudaStream_t st = (cudaStream_t)stream;
    n->t += 1;
    const float c1 = 1.0f - powf(beta1, (float)n->t), c2 = 1.0f - powf(beta2, (float)n->t);
    adam_kernel<<<(N_PARAMS + 255) / 256, 256, 0, st>>>(n->P, n->G, n->Mm, n->Vm, N_PARAMS, lr, beta1, beta2, eps, c1,
                                                         c2, mlp_copies(n));
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return abi_cuda_fail(n->ctx, e, "mlp adam");
    return CSV_OK;
}

int csv_mlp_status(const csv_mlp* n) {
    if (!n) return CSV_EINVAL;
    DeviceGuard g(n->ctx->device);
    uint32_t err = 0;
    if (cudaMemcpy(&err, n->err, 4, cudaMemcpyDeviceToHost) != cudaSuccess) return CSV_ECUDA;
    return err ? CSV_ECUDA : CSV_OK;
}

int csv_brick_features(csv_ctx* ctx, const uint64_t* d_volume, uint32_t W, uint32_t H, uint32_t D,
                       uint32_t brick_size, float* d_features, void* stream) {
    if (!ctx || !d_volume || !d_features) return CSV_EINVAL;
    if (brick_size < 8 || brick_size > 64 || (brick_size & (brick_size - 1)))
        return abi_fail(ctx, CSV_EINVAL, "features: brick size must be a power of two in [8, 64]");
    DeviceGuard g(ctx->device);
    const uint32_t nbx = (W + brick_size - 1) / brick_size, nby = (H + brick_size - 1) / brick_size,
                   nbz = (D + brick_size - 1) / brick_size;
    const uint64_t nb = (uint64_t)nbx * nby * nbz;
    if (nb == 0) return CSV_OK;
    // CTAs per brick: four rows or more per warp each, and no more than fill the device a few times over
    const uint32_t rows = (brick_size / 2) * (brick_size / 2);
    uint32_t parts = 1;
    while (2 * parts * 4 * (kFThreads / 32) <= rows && parts * nb < 2048) parts *= 2;
    cudaError_t e = cudaMemsetAsync(d_features, 0, nb * kFeat * sizeof(float), (cudaStream_t)stream);
    if (e == cudaSuccess) {
        features_kernel<<<(uint32_t)nb * parts, kFThreads, 0, (cudaStream_t)stream>>>(
            d_volume, W, H, D, brick_size, nbx, nby, nbz, parts, d_features);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) return abi_cuda_fail(ctx, e, "features");
    return CSV_OK;
}

int csv_encode_stats(csv_ctx* ctx, const uint64_t* d_volume, uint32_t W, uint32_t H, uint32_t D, uint32_t brick_size,
                     uint32_t* d_hist, void* stream) {
    if (!ctx || !d_volume || !d_hist) return CSV_EINVAL;
    if (brick_size < 8 || brick_size > 64 || (brick_size & (brick_size - 1)))
        return abi_fail(ctx, CSV_EINVAL, "brick size must be a power of two in [8, 64]");
    DeviceGuard g(ctx->device);
    if (!ctx->enc) ctx->enc = encoder_state_new();
    std::string err;
    int rc = encode_stats(ctx->enc, ctx->device, d_volume, W, H, D, brick_size, d_hist, (cudaStream_t)stream, err);
    if (rc) return abi_fail(ctx, rc, err);
    return CSV_OK;
}

int csv_select_exhaustive(csv_ctx* ctx, const uint32_t* d_hist, uint32_t n_bricks, const uint32_t* tables,
                          uint32_t n_tables, uint8_t* d_sel, uint64_t* d_cost, void* stream) {
    if (!ctx || !d_hist || !tables || !d_sel || n_tables == 0 || n_tables > kTablesN) return CSV_EINVAL;
    DeviceGuard g(ctx->device);
    // bits per symbol, 16.16 fixed point: -log2(f / 4096)
    CodeLengths len = {};
    for (uint32_t t = 0; t < n_tables; ++t)
        for (int s = 0; s < 16; ++s) {
            const uint32_t f = tables[t * 16 + s];
            if (f == 0 || f > kTot) return abi_fail(ctx, CSV_EINVAL, "select: table frequency out of range");
            len.v[t * 16 + s] = (uint32_t)llround(-log2((double)f / (double)kTot) * 65536.0);
        }
    cudaError_t e = cudaSuccess;
    if (n_bricks) {
        select_kernel<<<(n_bricks + kSelWarps - 1) / kSelWarps, 32 * kSelWarps, 0, (cudaStream_t)stream>>>(
            d_hist, n_bricks, len, n_tables, d_sel, d_cost);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize((cudaStream_t)stream);
    if (e != cudaSuccess) return abi_cuda_fail(ctx, e, "select");
    return CSV_OK;
}

int csv_encode_device_sel(csv_ctx* ctx, const uint64_t* d_volume, uint32_t W, uint32_t H, uint32_t D,
                          uint32_t brick_size, const uint32_t* tables, uint32_t n_tables, const uint8_t* d_sel,
                          void* stream, size_t* image_len) {
    if (!ctx || !d_volume || (n_tables && !tables) || n_tables > kTablesN) return CSV_EINVAL;
    if (brick_size < 8 || brick_size > 64 || (brick_size & (brick_size - 1)))
        return abi_fail(ctx, CSV_EINVAL, "brick size must be a power of two in [8, 64]");
    DeviceGuard g(ctx->device);
    if (!ctx->enc) ctx->enc = encoder_state_new();
    EncodeSelection sel;
    sel.n_tables = n_tables;
    for (uint32_t t = 0; t < n_tables; ++t)
        for (int s = 0; s < 16; ++s) sel.freq[t][s] = tables[t * 16 + s];
    sel.d_sel = d_sel;
    std::string err;
    int rc = encode_device(ctx->enc, ctx->device, d_volume, W, H, D, brick_size, (cudaStream_t)stream, err, &sel);
    if (rc) return abi_fail(ctx, rc, err);
    size_t len = 0;
    encoder_image(ctx->enc, &len);
    if (image_len) *image_len = len;
    return CSV_OK;
}

// ---- selector files: the fitted tables and the trained network, so that a
// learned encode needs no training run.  Little-endian: u32 magic "CSVS"
// (0x53565343), u32 version 1, u32 CSV_MLP_PARAMS, u32 n_tables (1..16), u32
// tables[n_tables][16], f32 params[CSV_MLP_PARAMS], u32 FNV-1a of every byte
// before it.
static uint32_t fnv1a(const uint8_t* p, size_t n, uint32_t h = 2166136261u) {
    for (size_t i = 0; i < n; ++i) h = (h ^ p[i]) * 16777619u;
    return h;
}
static bool tables_ok(const uint32_t* t, uint32_t n) {
    if (n == 0 || n > kTablesN) return false;
    for (uint32_t k = 0; k < n; ++k) {
        uint32_t sum = 0;
        for (int s = 0; s < 16; ++s) {
            if (t[k * 16 + s] == 0) return false;
            sum += t[k * 16 + s];
        }
        if (sum != kTot) return false;
    }
    return true;
}
constexpr uint32_t kSelMagic = 0x53565343u;

int csv_selector_write(const char* path, const float* params, const uint32_t* tables, uint32_t n_tables) {
    if (!path || !params || !tables) return CSV_EINVAL;
    if (!tables_ok(tables, n_tables)) return CSV_EINVAL;
    std::vector<uint8_t> buf;
    auto put = [&](const void* p, size_t n) {
        const uint8_t* b = (const uint8_t*)p;
        buf.insert(buf.end(), b, b + n);
    };
    const uint32_t head[4] = {kSelMagic, 1u, (uint32_t)N_PARAMS, n_tables};
    put(head, sizeof head);
    put(tables, 64ull * n_tables);
    put(params, 4ull * N_PARAMS);
    const uint32_t h = fnv1a(buf.data(), buf.size());
    put(&h, 4);
    FILE* f = fopen(path, "wb");
    if (!f) return CSV_EIO;
    const size_t w = fwrite(buf.data(), 1, buf.size(), f);
    const int c = fclose(f);
    return (w == buf.size() && c == 0) ? CSV_OK : CSV_EIO;
}

int csv_selector_read(const char* path, float* params, uint32_t* tables, uint32_t* n_tables) {
    if (!path || !params || !tables || !n_tables) return CSV_EINVAL;
    FILE* f = fopen(path, "rb");
    if (!f) return CSV_EIO;
    std::vector<uint8_t> buf;
    uint8_t tmp[65536];
    size_t r;
    while ((r = fread(tmp, 1, sizeof tmp, f)) > 0) buf.insert(buf.end(), tmp, tmp + r);
    fclose(f);
    if (buf.size() < 20) return CSV_EFORMAT;
    uint32_t head[4];
    memcpy(head, buf.data(), sizeof head);
    if (head[0] != kSelMagic || head[1] != 1u || head[2] != (uint32_t)N_PARAMS || head[3] == 0 || head[3] > kTablesN)
        return CSV_EFORMAT;
    const size_t need = 16 + 64ull * head[3] + 4ull * N_PARAMS + 4;
    if (buf.size() != need) return CSV_EFORMAT;
    uint32_t h;
    memcpy(&h, buf.data() + need - 4, 4);
    if (h != fnv1a(buf.data(), need - 4)) return CSV_EFORMAT;
    if (!tables_ok(reinterpret_cast<const uint32_t*>(buf.data() + 16), head[3])) return CSV_EFORMAT;
    memcpy(tables, buf.data() + 16, 64ull * head[3]);
    memcpy(params, buf.data() + 16 + 64ull * head[3], 4ull * N_PARAMS);
    *n_tables = head[3];
    return CSV_OK;
}

// The learned encode in one call: features of every brick, the network's
// choice, the encode with those choices into a version-2 image.
int csv_encode_learned(csv_ctx* ctx, const uint64_t* d_volume, uint32_t W, uint32_t H, uint32_t D,
                       uint32_t brick_size, csv_mlp* net, const uint32_t* tables, uint32_t n_tables, void* stream,
                       size_t* image_len) {
    if (!ctx || !d_volume || !net || !tables) return CSV_EINVAL;
    if (!tables_ok(tables, n_tables)) return abi_fail(ctx, CSV_EINVAL, "learned encode: tables must sum to 4096");
    if (brick_size < 8 || brick_size > 64 || (brick_size & (brick_size - 1)))
        return abi_fail(ctx, CSV_EINVAL, "brick size must be a power of two in [8, 64]");
    DeviceGuard g(ctx->device);
    const uint64_t nb = (uint64_t)((W + brick_size - 1) / brick_size) * ((H + brick_size - 1) / brick_size) *
                        ((D + brick_size - 1) / brick_size);
    if (nb == 0 || nb > 0xFFFFFFFFull) return abi_fail(ctx, CSV_ERANGE, "learned encode: brick count");
    float* d_feat = nullptr;
    uint8_t* d_sel = nullptr;
    // (from the context's pool: a plain allocation and its release map memory anew each time, 0.6 ms)
    cudaStream_t st = (cudaStream_t)stream;
    cudaError_t e = tmp_alloc((void**)&d_feat, nb * CSV_FEATURES * sizeof(float), ctx->pool, st);
    if (e == cudaSuccess) e = tmp_alloc((void**)&d_sel, nb, ctx->pool, st);
    if (e != cudaSuccess) {
        if (d_feat) cudaFreeAsync(d_feat, st);
        return abi_cuda_fail(ctx, e, "learned encode");
    }
    int rc = csv_brick_features(ctx, d_volume, W, H, D, brick_size, d_feat, stream);
    if (rc == CSV_OK) rc = csv_mlp_forward(net, d_feat, (uint32_t)nb, nullptr, d_sel, stream);
    if (rc == CSV_OK)
        rc = csv_encode_device_sel(ctx, d_volume, W, H, D, brick_size, tables, n_tables, d_sel, stream, image_len);
    cudaFreeAsync(d_feat, st);
    cudaFreeAsync(d_sel, st);
    cudaStreamSynchronize(st);
    return rc;
}

}  // extern "C"
