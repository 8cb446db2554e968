// encode.cu -- sm_100a brick encoder, byte-identical to the reference encoder.
//
// Reference behaviour restated here (paths relative to the reference root):
//   splitGridIntoBricks   brick.hpp:133-195     Brick::build       brick.hpp:78-123
//   majorityVote8         brick.hpp:24-37       bestOperation      brickEncoding.hpp:188-318
//   encodeBrick           brickEncoding.hpp:348-447
//   packOperationsToNibbles brickEncoding.cpp:11-91
//   updateFrequencyTables brickEncoding.cpp:94-144 (bricks i % 512 == 0, brickEncoding.hpp:481-482)
//   buildRansModel        brickEncoding.cpp:146-200
//   ransEncodeSymbol/ransFlush brickEncoding.cpp:202-219, brickEncoding.hpp:452-526
//   saveDatasetToFile     fileIO.cpp:15-99
//
// Pipeline (one launch each):
//   K1 enc_bricks: one CTA per brick (persistent).  Builds the majority pyramid
//      straight from the volume (no Morton-ordered copy of the leaves) and the
//      list of its non-constant nodes, chooses Rp/Rx/Ry/Rz for each of their
//      children in parallel, leaves the palette ops to one warp that walks them
//      in stream order with a 17-entry window of the most recent palette entries
//      (reverse find only matters up to distance 16: farther or absent means Pa),
//      then lays out nibbles with a block scan and packs them.  Also records, for
//      the seek index, the nibble and palette index of every S-th op.
//   K2 model: buildRansModel on the shared 16-bin histogram.
//   K3 rans: one chain per brick, symbols in reverse; while encoding it also
//      records the decoder state at the seek checkpoints (the decoder's state
//      before symbol i is the encoder's state after symbol i).
//   K4 serialize: header + records, file order.
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <string>
#include <type_traits>
#include <vector>

#include "block_scan.cuh"
#include "csv_internal.h"
#include "majority.cuh"

namespace csv {

constexpr uint32_t kEncSmemLevels = 5;  // levels 0..4 in shared memory
constexpr uint32_t OP_PALNEED = 7;  // placeholder code until the palette walk decides P0 / Pd / Pa
constexpr uint32_t EF_UNIFORM = 1u, EF_OVERFLOW = 2u;
// Encoder counters (u64 words): 0 nibble pool head, 1 palette pool head,
// 2..17 the sampled bricks' nibble histogram, 18 the brick work queue (low
// 32 bits), 19 checkpoint pool head, 20 stream pool head, 21 the image's length.
constexpr uint32_t kMiscQueue = 18, kMiscCk = 19, kMiscEnc = 20, kMiscImage = 21, kMiscWords = 32;
constexpr uint32_t kModes = 12;
constexpr uint32_t kMaxTables = 16;
constexpr uint32_t kModelWords = 65;  // freq[16] cum[16] total M[16] shift[16]

struct EncMeta {
    uint64_t nib_off, pal_off, enc_off;
    uint32_t P, nsym, nbytes, n_ops;
    uint32_t id, flags, n_ck, E;
    uint32_t level_start[8];
    uint32_t sel;     // mode | table << 4
    uint32_t ck_off;  // first of the brick's n_ck seek checkpoints in the checkpoint pool
};

struct EncoderState {
    int device = 0;
    uint32_t b = 0, L = 0, nb = 0, S = kOpsPerCheckpoint;
    uint64_t ck_used = 0;  // checkpoints of the last encode (pool entries in use)
    bool bricks_done = false;  // a shard's K1 ran; finish_encode_shard completes the image
    uint64_t W = 0, H = 0, D = 0;
    // buffers (grow-only)
    EncMeta* d_meta = nullptr;
    size_t meta_cap = 0;
    Checkpoint* d_ck = nullptr;
    size_t ck_cap_total = 0;
    uint8_t* d_nib = nullptr;
    size_t nib_cap = 0;
    uint64_t* d_pal = nullptr;
    size_t pal_cap = 0;
    uint8_t* d_enc = nullptr;
    size_t enc_cap = 0;
    uint64_t* d_rec_off = nullptr;
    size_t rec_cap = 0;
    uint64_t enc_need = 0;  // bytes of the stream pool that the last K1 gave out
    uint8_t* d_scratch = nullptr;
    size_t scratch_cap = 0;
    unsigned long long* d_misc = nullptr;  // [0] nib head, [1] pal head, [2..17] histogram, [18] queue
    uint32_t* d_model = nullptr;           // freq[16] cum[17] M[16] sh[16]
    uint8_t* d_image = nullptr;
    size_t image_cap = 0, image_len = 0;
    uint32_t freq[16] = {}, cum[17] = {};
    uint32_t n_tables = 1;                       // rANS models of the last image
    uint32_t tab_freq[16][16] = {}, tab_cum[16][16] = {};
    bool v2 = false;
    // page-locked: what an encode reads back
    EncMeta* h_meta = nullptr;
    size_t h_meta_cap = 0;
    struct Words {
        unsigned long long misc[kMiscWords];
        uint32_t model[kModelWords];
    }* h_words = nullptr;
    bool valid = false;
};

EncoderState* encoder_state_new() { return new EncoderState(); }

void encoder_state_free(EncoderState* s) {
    if (!s) return;
    cudaFree(s->d_meta);
    cudaFree(s->d_ck);
    cudaFree(s->d_nib);
    cudaFree(s->d_pal);
    cudaFree(s->d_enc);
    cudaFree(s->d_rec_off);
    cudaFree(s->d_scratch);
    cudaFree(s->d_misc);
    cudaFree(s->d_model);
    cudaFree(s->d_image);
    cudaFreeHost(s->h_meta);
    cudaFreeHost(s->h_words);
    delete s;
}

__device__ __forceinline__ uint32_t demorton_axis(uint32_t m) {
    m &= 0x09249249u;
    m = (m ^ (m >> 2)) & 0x030c30c3u;
    m = (m ^ (m >> 4)) & 0x0300f00fu;
    m = (m ^ (m >> 8)) & 0x030000ffu;
    m = (m ^ (m >> 16)) & 0x000003ffu;
    return m;
}
__device__ __forceinline__ uint32_t spread_axis(uint32_t v) {
    v &= 0x3ffu;
    v = (v | (v << 16)) & 0x030000ffu;
    v = (v | (v << 8)) & 0x0300f00fu;
    v = (v | (v << 4)) & 0x030c30c3u;
    v = (v | (v << 2)) & 0x09249249u;
    return v;
}
__device__ __forceinline__ uint32_t morton3(uint32_t x, uint32_t y, uint32_t z) {
    return spread_axis(x) | (spread_axis(y) << 1) | (spread_axis(z) << 2);
}

// ------------------------------------------------------------ K1 bricks
struct EncArgs {
    const uint64_t* vol;
    uint64_t W, H, D;
    uint32_t b, L, nbx, nby, nbz, nb;
    uint8_t* scratch;
    uint64_t scratch_per_cta;
    EncMeta* meta;
    uint8_t* nib_pool;
    uint64_t nib_cap;
    uint64_t* pal_pool;
    uint64_t pal_cap;
    Checkpoint* ck;     // checkpoint pool, reserved per brick at misc[kMiscCk]
    uint64_t ck_cap;    // pool entries
    uint32_t bx0;         // brick-x offset of this volume in a larger one (brick IDs)
    uint32_t index_base;  // file index of brick 0 in the larger volume (the model's sample rule)
    unsigned long long* misc;
    const uint8_t* sel;  // per brick: mode | table << 4 (null: mode 0, table 0)
    bool pairs;          // voxels 2k, 2k + 1 of a row are a 16-byte aligned pair
};

// Nodes and activity words of the levels: level l has 8^l nodes from lvl_off(l) on and
// one bit per node (set: the node is not constant, so its children have ops) in words
// from moff(l) on.
__host__ __device__ constexpr uint32_t lvl_off(uint32_t l) { return ((1u << (3 * l)) - 1) / 7; }
__host__ __device__ constexpr uint32_t mwords(uint32_t l) { return l < 2 ? 1u : (1u << (3 * l)) / 32; }
__host__ __device__ constexpr uint32_t moff(uint32_t l) { return l < 2 ? l : 2 + (lvl_off(l) - 9) / 32; }
static_assert(moff(2) == 2 && moff(3) == 4 && moff(5) == 148 && moff(6) == 1172, "one word below 32 nodes");

// A level's labels lie in raster order (x fastest, l bits an axis), so that neighbours are
// an addition away; its activity bits and its ops in Morton order, the stream's.
//
// A block's shared memory: fixed part, then the labels of levels 0 .. min(L - 2, 4), the
// activity words of levels 0 .. L - 2, then staging.
struct EncFixed {
    uint32_t sh32[33];
    uint32_t hist[64];
    uint32_t level_r[8];  // active nodes before level l's, l = 0 .. L - 1
    uint32_t work, P, n_pd, n_act;
    uint64_t nib_off, pal_off, ck_off, enc_off;
};
__host__ __device__ inline uint32_t enc_lab_nodes(uint32_t L) {
    return lvl_off(L - 1 < kEncSmemLevels ? L - 1 : kEncSmemLevels);
}
template <int T>
__host__ __device__ inline uint32_t enc_smem(uint32_t L) {
    const uint32_t lab = (8 * enc_lab_nodes(L) + 15) & ~15u, nw = (moff(L - 1) + 7) & ~7u;
    return lab + 4 * nw + T * 16 + 32;
}
// Active nodes whose palette ops the walk lists at a time (their ops numbered in 16 bits).
template <int T>
constexpr uint32_t kWalkParents = T * 16 * 8 <= 65536 ? T * 16 : 8192;
// A block's scratch in global memory (it stays in L2).
struct EncScratch {
    uint64_t lab, ops, need8, act, pal, bytes;  // offsets, and all of it
};
template <int T>
__host__ __device__ inline EncScratch enc_scratch(uint32_t L) {
    const uint64_t max_ops = ((1ull << (3 * L)) - 8) / 7, max_act = lvl_off(L - 1);
    auto align = [](uint64_t v) { return (v + 255) & ~255ull; };
    // the walk's list of a block's worth of parents takes the active nodes' place
    const uint64_t list = 2 * 8 * (max_act < kWalkParents<T> ? max_act : kWalkParents<T>);
    EncScratch X;
    X.lab = 0;
    X.ops = L >= kEncSmemLevels + 2 ? align(8ull << (3 * (L - 2))) : 0;
    X.need8 = align(X.ops + max_ops + 16);
    X.act = align(X.need8 + max_act + 16);
    X.pal = align(X.act + (4 * max_act > list ? 4 * max_act : list));
    X.bytes = align(X.pal + 8 * max_ops);
    return X;
}

struct BrickCtx {
    const EncArgs* A;
    EncFixed* S;
    uint64_t* lab;   // shared: labels of levels 0 .. 4
    uint32_t* mask;  // shared: activity words
    uint8_t* room;   // shared: staging (before: the pyramid's queues)
    uint64_t* lab_g;  // scratch: labels of level 5
    uint8_t* ops;     // scratch: code | stop << 3 | delta << 4, in stream order
    uint8_t* need8;   // scratch: per active node, which of its children take a palette op
    uint32_t* act;    // scratch: the active nodes in stream order, raster | Morton << 16
    uint64_t* pal_lab;  // scratch: the labels of the ops that do; the palette from its start on
    const uint64_t* vol;  // the brick's first voxel
    uint64_t WH;
    uint32_t x_lim, y_lim, z_lim;  // voxels of the brick inside the volume
    bool interior;
};

__device__ __forceinline__ uint64_t voxel(const BrickCtx& B, uint32_t x, uint32_t y, uint32_t z) {
    if (B.interior || (x < B.x_lim && y < B.y_lim && z < B.z_lim))
        return __ldg(B.vol + (x + B.A->W * y + B.WH * z));
    return 0;  // padding, brick.hpp:181-183
}
// The eight voxels of node (x, y, z) of the level above the leaves; as 16-byte pairs
// along x when the volume's rows hold them aligned.
__device__ __forceinline__ void voxels8(const BrickCtx& B, uint32_t x, uint32_t y, uint32_t z, uint64_t v[8]) {
    if (B.interior && B.A->pairs) {
        const uint64_t* p = B.vol + (2 * x + B.A->W * (2 * y) + B.WH * (2 * z));
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const ulonglong2 t =
                __ldg(reinterpret_cast<const ulonglong2*>(p + ((r & 1) ? B.A->W : 0) + ((r & 2) ? B.WH : 0)));
            v[2 * r] = t.x;
            v[2 * r + 1] = t.y;
        }
    } else {
#pragma unroll
        for (int c = 0; c < 8; ++c) v[c] = voxel(B, 2 * x + (c & 1), 2 * y + ((c >> 1) & 1), 2 * z + (c >> 2));
    }
}

// Decoder-transparent encoding modes.  Where several ops reproduce a child's
// label, bestOperation (brickEncoding.hpp:198-282) takes Rp, then Rx, Ry, Rz,
// then a palette op.  A mode keeps the grammar and changes that preference:
// mode % 6 picks the order of the three neighbour axes, and modes >= 6 try the
// neighbours before the parent.  The decoder replays any of them unchanged;
// mode 0 is the reference's order.
// mode_codes(m): the op code for each set of matches (bit 0 the parent, bits 1..3 the
// neighbours along x, y, z), 3 bits per set; none: a palette op.
__host__ __device__ constexpr uint64_t mode_codes(uint32_t mode) {
    const uint32_t order[6] = {012, 021, 0102, 0120, 0201, 0210};  // axes, first one on top (octal digits)
    uint64_t t = 0;
    for (uint32_t set = 0; set < 16; ++set) {
        uint32_t code = OP_PALNEED;
        for (uint32_t k = 0; k < 3 && code == OP_PALNEED; ++k) {
            const uint32_t a = (order[mode % 6] >> (3 * (2 - k))) & 7u;
            if ((set >> (a + 1)) & 1u) code = OP_RX + a;
        }
        if ((set & 1u) && (mode < 6 || code == OP_PALNEED)) code = OP_RP;
        t |= (uint64_t)code << (3 * set);
    }
    return t;
}
struct ModeTable {
    uint64_t t[kModes];
};
constexpr ModeTable make_mode_table() {
    ModeTable m{};
    for (uint32_t k = 0; k < kModes; ++k) m.t[k] = mode_codes(k);
    return m;
}
__constant__ ModeTable kModeTable = make_mode_table();

// The block's scratch and shared memory.
template <int T>
__device__ __forceinline__ BrickCtx enc_ctx(const EncArgs& A, EncFixed& S, uint8_t* smem) {
    uint8_t* scr = A.scratch + (uint64_t)blockIdx.x * A.scratch_per_cta;
    const EncScratch X = enc_scratch<T>(A.L);
    const uint32_t nw = (moff(A.L - 1) + 7) & ~7u;
    BrickCtx B;
    B.A = &A;
    B.S = &S;
    B.lab = reinterpret_cast<uint64_t*>(smem);
    smem += (8 * enc_lab_nodes(A.L) + 15) & ~15u;
    B.mask = reinterpret_cast<uint32_t*>(smem);
    B.room = smem + 4 * nw;
    B.lab_g = reinterpret_cast<uint64_t*>(scr + X.lab);
    B.ops = scr + X.ops;
    B.need8 = scr + X.need8;
    B.act = reinterpret_cast<uint32_t*>(scr + X.act);
    B.pal_lab = reinterpret_cast<uint64_t*>(scr + X.pal);
    B.WH = A.W * A.H;
    return B;
}

// Brick i (split order: bx outer, bz inner, brick.hpp:152-154).
__device__ __forceinline__ void enc_place(BrickCtx& B, uint32_t bx, uint32_t by, uint32_t bz) {
    const EncArgs& A = *B.A;
    const uint64_t x0 = (uint64_t)bx * A.b, y0 = (uint64_t)by * A.b, z0 = (uint64_t)bz * A.b;
    B.vol = A.vol + (x0 + A.W * (y0 + A.H * z0));
    B.x_lim = (uint32_t)min(A.W - x0, (uint64_t)A.b);
    B.y_lim = (uint32_t)min(A.H - y0, (uint64_t)A.b);
    B.z_lim = (uint32_t)min(A.D - z0, (uint64_t)A.b);
    B.interior = B.x_lim == A.b && B.y_lim == A.b && B.z_lim == A.b;
}

// Position of the k-th set bit of b (k below its number of set bits).
__device__ __forceinline__ uint32_t nth_bit(uint32_t b, uint32_t k) {
    uint32_t at = 0;
#pragma unroll
    for (uint32_t h = 16; h; h >>= 1) {
        const uint32_t low = __popc((b >> at) & ((1u << h) - 1u));
        if (k >= low) {
            k -= low;
            at += h;
        }
    }
    return at;
}

// The list of the active nodes (B.act) and S.level_r from the activity words; returns
// their number.  A warp takes 32 words at a time and gives every lane one of their set
// bits.  Every thread of the block calls it.
template <int T>
__device__ uint32_t list_active(const BrickCtx& B) {
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, L = B.A->L, FULL = 0xFFFFFFFFu;
    const uint32_t nw = moff(L - 1), n_grp = (nw + 31) / 32;  // at most 37 groups of words
    uint32_t* sum = B.S->hist;  // per group: active nodes, then those before it
    for (uint32_t g = warp; g < n_grp; g += T / 32) {
        const uint32_t w = 32 * g + lane;
        const uint32_t n = __reduce_add_sync(FULL, w < nw ? __popc(B.mask[w]) : 0u);
        if (lane == 0) sum[g] = n;
    }
    __syncthreads();
    if (warp == 0) {
        const uint32_t a = 2 * lane < n_grp ? sum[2 * lane] : 0u, b = 2 * lane + 1 < n_grp ? sum[2 * lane + 1] : 0u;
        uint32_t inc = a + b;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL, inc, d);
            if (lane >= (uint32_t)d) inc += y;
        }
        sum[2 * lane] = inc - a - b;
        sum[2 * lane + 1] = inc - b;
        if (lane == 31) B.S->n_act = inc;
    }
    __syncthreads();
    for (uint32_t g = warp; g < n_grp; g += T / 32) {
        const uint32_t w = 32 * g + lane, bits = w < nw ? B.mask[w] : 0u, cnt = __popc(bits);
        uint32_t inc = cnt;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL, inc, d);
            if (lane >= (uint32_t)d) inc += y;
        }
        const uint32_t base = sum[g], total = __shfl_sync(FULL, inc, 31);
        uint32_t l = 0;  // the word's level
#pragma unroll
        for (uint32_t k = 1; k < 6; ++k) l += w >= moff(k) ? 1u : 0u;
        if (w < nw && w == moff(l)) B.S->level_r[l] = base + inc - cnt;
        for (uint32_t t0 = 0; t0 < total; t0 += 32) {
            const uint32_t t = t0 + lane;
            uint32_t j = 0;  // the lane whose word has the t-th node: as many as end at or before t
#pragma unroll
            for (uint32_t h = 16; h; h >>= 1)
                if (__shfl_sync(FULL, inc, j + h - 1) <= t) j += h;
            j = min(j, 31u);
            const uint32_t wb = __shfl_sync(FULL, bits, j), before = __shfl_sync(FULL, inc - cnt, j),
                           wl = __shfl_sync(FULL, l, j);
            if (t < total) {
                const uint32_t m = 32 * (32 * g + j - moff(wl)) + nth_bit(wb, t - before);
                B.act[base + t] = demorton_axis(m) | demorton_axis(m >> 1) << wl | demorton_axis(m >> 2) << (2 * wl) |
                                  m << 16;
            }
        }
    }
    if (tid < 8 && tid >= L - 1) B.S->level_r[tid] = B.S->n_act;
    __syncthreads();
    return B.S->n_act;
}

// The majority pyramid of one brick (Brick::build, brick.hpp:78-123) and its active
// nodes.  Returns their number.  Most nodes above the leaves hold one label, so a warp
// first only tells which do (32 nodes in raster order at a time, so that it reads whole
// rows of the brick: rows of 64 bytes, as 32 Morton-consecutive nodes have them, ran at
// 0.7 of the rate); the others it queues, and takes the vote over 32 of them at once.
template <int T>
__device__ uint32_t build_pyramid(const BrickCtx& B) {
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, L = B.A->L, lb = L - 2;
    const uint32_t sm = (1u << lb) - 1u, FULL = 0xFFFFFFFFu;
    uint64_t* lab = lb < kEncSmemLevels ? B.lab + lvl_off(lb) : B.lab_g;
    uint16_t* queue = reinterpret_cast<uint16_t*>(B.room) + 64 * warp;
    for (uint32_t w = tid; w < mwords(lb); w += T) B.mask[moff(lb) + w] = 0;
    __syncthreads();
    uint32_t queued = 0;
    auto vote = [&](uint32_t n) {  // of the first n queued
        if (lane < n) {
            const uint32_t p = queue[lane];
            uint64_t v[8];
            voxels8(B, p & sm, (p >> lb) & sm, p >> (2 * lb), v);
            lab[p] = majority8_mixed(v);
        }
        __syncwarp();
    };
    for (uint32_t w = warp; w < mwords(lb); w += T / 32) {
        const uint32_t p = 32 * w + lane;
        bool active = false;
        if (p < 1u << (3 * lb)) {
            uint64_t v[8];
            voxels8(B, p & sm, (p >> lb) & sm, p >> (2 * lb), v);
            active = !uniform8(v);
            if (!active) lab[p] = v[0];
        }
        const uint32_t bits = __ballot_sync(FULL, active);
        if (!bits) continue;
        // the activity bits in Morton order: four consecutive x of one (y, z) are bits 0, 1, 8, 9 from
        // the row's place in their word on (levels of fewer nodes: the first of them)
        const uint32_t four = (bits >> (4 * (lane & 7u))) & 15u;
        if (lane < 8 && four) {
            const uint32_t q = 32 * w + 4 * lane;
            if (lb >= 2) {
                const uint32_t m = morton3(q & sm, (q >> lb) & sm, q >> (2 * lb));
                atomicOr(B.mask + moff(lb) + (m >> 5), ((four & 3u) | (four & 12u) << 6) << (m & 31u));
            } else {  // at most 2 x 2 x 2 nodes: both orders are one
                atomicOr(B.mask + moff(lb), four << (4 * lane));
            }
        }
        if (active) queue[queued + __popc(bits & ((1u << lane) - 1u))] = (uint16_t)p;
        queued += __popc(bits);
        __syncwarp();
        if (queued >= 32) {
            vote(32);
            queued -= 32;
            if (lane < queued) queue[lane] = queue[32 + lane];
            __syncwarp();
        }
    }
    vote(queued);
    __syncthreads();
    for (int l = (int)lb - 1; l >= 0; --l) {  // buildLevel (brick.hpp:92-123)
        const uint64_t* below = l + 1 < (int)kEncSmemLevels ? B.lab + lvl_off(l + 1) : B.lab_g;
        for (uint32_t w = warp; w < mwords(l); w += T / 32) {
            const uint32_t m = 32 * w + lane;
            bool active = false;
            if (m < 1u << (3 * l)) {
                const uint32_t x = demorton_axis(m), y = demorton_axis(m >> 1), z = demorton_axis(m >> 2);
                const uint32_t first = 2 * x | (2 * y) << (l + 1) | (2 * z) << (2 * l + 2);
                uint64_t v[8];
#pragma unroll
                for (int r = 0; r < 4; ++r) {  // (one voxel's level is a single, so 8-byte aligned, label)
                    const uint64_t* q = below + (first | (r & 1) << (l + 1) | (r >> 1) << (2 * l + 2));
                    v[2 * r] = q[0];
                    v[2 * r + 1] = q[1];
                }
                bool all;
                B.lab[lvl_off(l) + (x | y << l | z << (2 * l))] = majority8(v, all);
                // active when a child is, or when the children differ
                active = !all || ((B.mask[moff(l + 1) + (m >> 2)] >> (8 * (m & 3u))) & 0xFFu) != 0;
            }
            const uint32_t bits = __ballot_sync(FULL, active);
            if (lane == 0) B.mask[moff(l) + w] = bits;
        }
        __syncthreads();
    }
    return list_active<T>(B);
}

// The ops of the children of level l's active nodes (encodeBrick, brickEncoding.hpp:372-433):
// the r-th active node's (levels in order, Morton order within a level) are ops 8r .. 8r +
// 7.  A warp takes four active nodes at a time, a child per lane.  f(r, c, set, stop,
// label): which of the parent (bit 0) and the neighbours outside the sibling block (bits
// 1 .. 3) have the child's label (bestOperation, :198-282; all of them when `every`, else
// the neighbours only where the parent has not), for every lane of the warp (stop: 2
// where the lane has no child).  PG, CG: the level's own labels and its children's are
// level 5's, in scratch; LEAF: the children are voxels.
template <int T, bool PG, bool CG, bool LEAF, class F>
__device__ __forceinline__ void level_children(const BrickCtx& B, uint32_t l, bool every, F& f) {
    const uint32_t lane = threadIdx.x & 31, c = lane & 7u, g = lane >> 3, lc = l + 1, sm = (1u << l) - 1u;
    const uint32_t r0 = B.S->level_r[l], n = B.S->level_r[l + 1] - r0;
    const uint32_t* act = B.act + r0;
    const uint64_t* lab_p = PG ? B.lab_g : B.lab + lvl_off(l);
    const uint64_t* lab_c = CG ? B.lab_g : B.lab + lvl_off(lc);  // (not used for leaves)
    const uint64_t W = B.A->W;
    auto child = [&](uint32_t p, uint32_t& x, uint32_t& y, uint32_t& z) {
        x = 2 * (p & sm) | (c & 1u);
        y = 2 * ((p >> l) & sm) | ((c >> 1) & 1u);
        z = 2 * (p >> (2 * l)) | (c >> 2);
    };
    // the nodes two steps ahead and the labels one step ahead are on their way
    uint32_t k = 4 * (threadIdx.x >> 5) + g;
    auto load_e = [&](uint32_t i) { return i < n ? act[i] : 0u; };
    auto load_labels = [&](uint32_t i, uint32_t e, uint64_t& parent, uint64_t& label) {
        parent = label = 0;
        if (i >= n) return;
        const uint32_t p = e & 0xFFFFu;
        uint32_t x, y, z;
        child(p, x, y, z);
        parent = lab_p[p];
        if (!LEAF) label = lab_c[x | y << lc | z << (2 * lc)];
        else if (B.interior || (x < B.x_lim && y < B.y_lim && z < B.z_lim)) label = __ldg(B.vol + (x + W * y + B.WH * z));
    };
    uint32_t e_next = load_e(k), e_after = load_e(k + T / 8);
    uint64_t parent_next, label_next;
    load_labels(k, e_next, parent_next, label_next);
    for (uint32_t q = k - g; q < n; q += T / 8, k += T / 8) {
        const uint32_t e = e_next;
        const uint64_t parent = parent_next, label = label_next;
        e_next = e_after;
        e_after = load_e(k + T / 4);
        load_labels(k + T / 8, e_next, parent_next, label_next);
        uint32_t set = 0, stop = 2;
        if (k < n) {
            const uint32_t p = e & 0xFFFFu, m = e >> 16;
            stop = LEAF ? 1u  // leaves are constant (brick.hpp:188)
                        : ((B.mask[moff(lc) + (m >> 2)] >> (8 * (m & 3u) + c)) & 1u ? 0u : 1u);
            set = parent == label ? 1u : 0u;
            if (every || !set) {
                uint32_t x, y, z;
                child(p, x, y, z);
                uint64_t nb[3];
                bool has[3];
#pragma unroll
                for (uint32_t a = 0; a < 3; ++a) {
                    const uint32_t at = (a == 0 ? x : (a == 1 ? y : z)) >> 1;
                    const bool up = (c >> a) & 1u;
                    has[a] = up ? at < sm : at > 0;
                    nb[a] = 0;
                    if (!has[a]) continue;
                    if (up) {  // +1 side: later in Morton order -> the neighbour's parent (:265-272)
                        nb[a] = lab_p[p + (1u << (a * l))];
                    } else if (!LEAF) {  // -1 side: earlier in Morton order -> the neighbour itself (:256-261)
                        nb[a] = lab_c[(x | y << lc | z << (2 * lc)) - (1u << (a * lc))];
                    } else {
                        nb[a] = voxel(B, x - (a == 0), y - (a == 1), z - (a == 2));
                    }
                }
#pragma unroll
                for (uint32_t a = 0; a < 3; ++a) set |= (has[a] && nb[a] == label ? 2u : 0u) << a;
            }
        }
        f(r0 + k, c, set, stop, label);
    }
}
template <int T, class F>
__device__ __forceinline__ void for_children(const BrickCtx& B, bool every, F f) {
    const uint32_t lb = B.A->L - 2;
    // the many first
    if (lb < kEncSmemLevels) level_children<T, false, false, true>(B, lb, every, f);
    else level_children<T, true, false, true>(B, lb, every, f);
    for (int l = (int)lb - 1; l >= 0; --l) {
        if (l + 1 < (int)kEncSmemLevels) level_children<T, false, false, false>(B, l, every, f);
        else level_children<T, false, true, false>(B, l, every, f);
    }
}

// Palette ops: the ops that need one are listed in stream order (8 or 16 active nodes
// per thread at a time), then the first warp takes them, 32 at a time, with a 17-entry
// window of the most recent palette entries (reverse find only matters up to distance 16:
// farther or absent means Pa).  The entries of a window differ, and only a miss changes
// it (the missed label enters at distance 0, the others move one on), so all 32 look
// their labels up at once and what is left to do in order is one step per miss.  put(j,
// code, delta) for every such op; the palette after the root's label goes to the start of
// pal_lab (an entry's place is never past that of an op still to come), its size to S.P
// and the number of Pd ops to S.n_pd.
template <int T, class F>
__device__ void palette_walk(const BrickCtx& B, uint64_t root, uint32_t n_act, F put) {
    const uint32_t tid = threadIdx.x, lane = tid & 31, FULL = 0xFFFFFFFFu;
    uint16_t* list = reinterpret_cast<uint16_t*>(B.act);  // (the active nodes' list is done with)
    uint64_t win = lane == 0 ? root : 0;
    uint32_t P = 1, n_pd = 0;
    constexpr uint32_t kPer = kWalkParents<T> / T;  // nodes per thread, 16 or 8
    static_assert(kPer * T == kWalkParents<T> && kPer % 4 == 0, "whole words of nodes per thread");
    for (uint32_t r0 = 0; r0 < n_act; r0 += kWalkParents<T>) {
        const uint32_t r = r0 + kPer * tid;
        uint32_t words[kPer / 4], cnt = 0;
#pragma unroll
        for (uint32_t q = 0; q < kPer / 4; ++q) {
            const uint32_t at = r + 4 * q;  // bytes below n_act
            words[q] = at < n_act ? *reinterpret_cast<const uint32_t*>(B.need8 + at) : 0u;
            if (at < n_act && at + 4 > n_act) words[q] &= (1u << (8 * (n_act - at))) - 1u;
            cnt += __popc(words[q]);
        }
        uint32_t total;
        uint32_t at = block_exclusive<uint32_t>(cnt, B.S->sh32, &total);
#pragma unroll
        for (uint32_t q = 0; q < kPer / 4; ++q)
            for (uint32_t m = words[q]; m; m &= m - 1)
                list[at++] = (uint16_t)(8 * kPer * tid + 32 * q + __ffs(m) - 1);
        __syncthreads();
        if (tid < 32 && total) {
            uint32_t j_next = lane < total ? 8 * r0 + list[lane] : 0u;
            uint64_t label_next = lane < total ? B.pal_lab[j_next] : 0ull;
            for (uint32_t k0 = 0; k0 < total; k0 += 32) {
                const bool valid = k0 + lane < total;
                const uint32_t j = j_next;
                const uint64_t mine = label_next;
                if (k0 + 32 + lane < total) {
                    j_next = 8 * r0 + list[k0 + 32 + lane];
                    label_next = B.pal_lab[j_next];
                }
                int d = -1;  // distance from the last entry
                const uint32_t depth = min(P, 17u);
                for (uint32_t k = 0; k < depth; ++k)
                    if (__shfl_sync(FULL, win, k) == mine) d = (int)k;
                bool added = false;
                for (uint32_t miss = __ballot_sync(FULL, valid && d < 0); miss;) {
                    const uint32_t f = __ffs(miss) - 1;
                    const uint64_t entry = __shfl_sync(FULL, mine, f), up = __shfl_up_sync(FULL, win, 1);
                    win = lane == 0 ? entry : up;
                    if (lane == 0) B.pal_lab[P - 1] = entry;
                    ++P;
                    if (lane == f) added = true;
                    if (lane > f) d = mine == entry ? 0 : (d >= 0 && d < 16 ? d + 1 : -1);
                    miss = __ballot_sync(FULL, valid && lane > f && d < 0);
                }
                const bool pd = valid && !added && d > 0;
                if (valid) put(j, added ? OP_PA : (d == 0 ? OP_P0 : OP_PD), pd ? (uint32_t)d - 1 : 0u);
                n_pd += __popc(__ballot_sync(FULL, pd));
            }
        }
        __syncthreads();
    }
    if (tid == 0) {
        B.S->P = P;
        B.S->n_pd = n_pd;
    }
    __syncthreads();
}

// Per byte of v whose op code is `code`: bit 0.
__device__ __forceinline__ uint32_t bytes_with(uint32_t v, uint32_t code) {
    const uint32_t x = (v & 0x07070707u) ^ (code * 0x01010101u);
    return ~(x | (x >> 1) | (x >> 2)) & 0x01010101u;
}
// Four op bytes as nibbles (op << 1 | stop, brickEncoding.cpp:66-67), the first lowest.
__device__ __forceinline__ uint32_t nibbles4(uint32_t v) {
    uint32_t n = ((v & 0x07070707u) << 1) | ((v >> 3) & 0x01010101u);
    n = (n | (n >> 4)) & 0x00FF00FFu;
    return (n | (n >> 8)) & 0xFFFFu;
}

// Bound by the volume's reads and their latency: the pyramid streams it (about two thirds
// of the HBM rate while every brick does so), the children's second look at the voxels of
// active nodes comes in pieces of 16 bytes.  Measured (B200) against a thread per run of
// nodes at every step and a palette walk over every op (two CTAs of 512 threads per SM):
// 512 bricks of 64^3 4.05 -> 0.76 ms (0.16 ms at the HBM rate), 8192 bricks of 32^3 3.33 ->
// 0.66 ms (0.32 ms), 60 bricks of 32^3 0.184 -> 0.054 ms.
template <int T, int PER_SM>
__global__ void __launch_bounds__(T, PER_SM) enc_bricks_kernel(EncArgs A) {
    extern __shared__ __align__(16) uint8_t enc_dyn[];
    __shared__ EncFixed S;
    const uint32_t tid = threadIdx.x;
    BrickCtx B = enc_ctx<T>(A, S, enc_dyn);
    for (;;) {
        if (tid == 0) S.work = atomicAdd(reinterpret_cast<unsigned int*>(A.misc + kMiscQueue), 1u);
        __syncthreads();
        const uint32_t i = S.work;
        if (i >= A.nb) break;
        const uint32_t bz = i % A.nbz, by = (i / A.nbz) % A.nby, bx = i / (A.nbz * A.nby);
        enc_place(B, bx, by, bz);
        const uint32_t sel = A.sel ? A.sel[i] : 0u, mode = min(sel & 15u, kModes - 1);
        const uint32_t n_act = build_pyramid<T>(B), n_ops = 8 * n_act;
        const uint64_t root = B.lab[0], codes = kModeTable.t[mode];
        for_children<T>(B, mode >= 6, [&](uint32_t r, uint32_t c, uint32_t set, uint32_t stop, uint64_t label) {
            const uint32_t code = (uint32_t)(codes >> (3 * set)) & 7u;
            const bool need = stop < 2 && code == OP_PALNEED;
            const uint32_t needs = __ballot_sync(0xFFFFFFFFu, need);
            if (stop < 2) {
                B.ops[8 * r + c] = (uint8_t)(code | stop << 3);
                if (need) B.pal_lab[8 * r + c] = label;
                if (c == 0) B.need8[r] = (uint8_t)(needs >> (threadIdx.x & 24u));
            }
        });
        __syncthreads();
        palette_walk<T>(B, root, n_act, [&](uint32_t j, uint32_t code, uint32_t delta) {
            B.ops[j] = (uint8_t)(code | (B.ops[j] & 8u) | delta << 4);
        });

        // ---- nibble layout (packOperationsToNibbles) and seek checkpoints
        const uint32_t P = S.P, nsym = 1 + n_ops + S.n_pd, nbytes = (nsym + 1) / 2;
        static_assert(kOpsPerCheckpoint == 16, "a thread's 16 ops start at a checkpoint");
        const uint32_t n_ck = (n_ops + 15) / 16;
        if (tid == 0) {
            S.ck_off = atomicAdd(A.misc + kMiscCk, (unsigned long long)n_ck);
            S.nib_off = atomicAdd(A.misc + 0, (unsigned long long)((nbytes + 15) & ~15u));
            S.pal_off = atomicAdd(A.misc + 1, (unsigned long long)P);
            // its stream: <= 2 bytes per symbol + flush
            S.enc_off = atomicAdd(A.misc + kMiscEnc, (4ull * nbytes + 4 + 15) & ~15ull);
        }
        if (tid < 16) S.hist[tid] = 0;
        // staging: packed nibbles from position `base` (a multiple of 32) on, nibble k at bit 4 k
        uint32_t* stage = reinterpret_cast<uint32_t*>(B.room);
        for (uint32_t k = tid; k < T * 4 + 8; k += T) stage[k] = 0;
        __syncthreads();
        const uint64_t nib_off = S.nib_off, pal_off = S.pal_off, ck_off = S.ck_off;
        const bool ck_ok = ck_off + n_ck <= A.ck_cap;
        // the rANS kernel reads whole 16-byte chunks of the reservation
        const bool ok = nib_off + ((nbytes + 15) & ~15u) <= A.nib_cap && pal_off + P <= A.pal_cap && ck_ok;
        const bool root_const = n_act == 0;
        const bool sample = ((A.index_base + i) % 512) == 0;  // brickEncoding.hpp:482
        Checkpoint* ck = A.ck + ck_off;
        uint4* nib = reinterpret_cast<uint4*>(A.nib_pool + nib_off);
        if (tid == 0) stage[0] = (OP_PA << 1) | (root_const ? 1u : 0u);
        uint32_t base = 0, pos = 1, pa = 0;  // the first position staged, the next one's, Pa ops before it
        // 16-byte chunk q of the staging, as the pool holds it (a byte's high nibble is the earlier one)
        auto chunk_out = [&](uint32_t q) {
            uint4 v = reinterpret_cast<const uint4*>(stage)[q];
            if (sample) {  // every nibble of the packed bytes, pad included (brickEncoding.cpp:131-143)
                uint64_t c[2] = {0, 0};
                const uint32_t words[4] = {v.x, v.y, v.z, v.w}, first = base + 32 * q;
#pragma unroll
                for (uint32_t k = 0; k < 32; ++k) {
                    const uint32_t s = (words[k >> 3] >> (4 * (k & 7u))) & 15u;
                    if (first + k < 2 * nbytes) (s & 8u ? c[1] : c[0]) += 1ull << (8 * (s & 7u));
                }
#pragma unroll
                for (uint32_t s = 0; s < 16; ++s) {
                    const uint32_t n = (uint32_t)(c[s >> 3] >> (8 * (s & 7u))) & 0xFFu;
                    if (n) atomicAdd(&S.hist[s], n);
                }
            }
            auto swap = [](uint32_t x) { return ((x & 0x0F0F0F0Fu) << 4) | ((x >> 4) & 0x0F0F0F0Fu); };
            if (ok) nib[base / 32 + q] = make_uint4(swap(v.x), swap(v.y), swap(v.z), swap(v.w));
        };
        for (uint32_t j0 = 0; j0 < n_ops; j0 += 16 * T) {
            const uint32_t j = j0 + 16 * tid;
            uint4 v = make_uint4(0, 0, 0, 0);
            uint32_t nv = 0;  // 16, or 8 at the end
            if (j < n_ops) {
                v = *reinterpret_cast<const uint4*>(B.ops + j);
                nv = min(16u, n_ops - j);
                if (nv == 8) v.z = v.w = 0;
            }
            const uint32_t d0 = bytes_with(v.x, OP_PD), d1 = bytes_with(v.y, OP_PD), d2 = bytes_with(v.z, OP_PD),
                           d3 = bytes_with(v.w, OP_PD);
            const uint32_t n_d = __popc(d0 | d1 << 1 | d2 << 2 | d3 << 3);
            const uint32_t n_a = __popc(bytes_with(v.x, OP_PA) | bytes_with(v.y, OP_PA) << 1 |
                                        bytes_with(v.z, OP_PA) << 2 | bytes_with(v.w, OP_PA) << 3);
            uint32_t total;
            const uint32_t before = block_exclusive<uint32_t>((nv + n_d) | n_a << 16, S.sh32, &total);
            const uint32_t at = pos + (before & 0xFFFFu);
            if (nv && ck_ok) ck[j >> 4] = Checkpoint{0, 0, at, pa + (before >> 16)};
            // the ops' nibbles into the staged words (neighbours share a word)
            uint32_t s = at - base;
            auto put = [&](uint64_t n) {  // up to 16 nibbles at s, zero above the last one
                const uint32_t sh = 4 * (s & 7u), k = s >> 3;
                const uint32_t lo = (uint32_t)n, hi = (uint32_t)(n >> 32);
                if (lo << sh) atomicOr(stage + k, lo << sh);
                const uint32_t mid = __funnelshift_l(lo, hi, sh), top = __funnelshift_l(hi, 0u, sh);
                if (mid) atomicOr(stage + k + 1, mid);
                if (top) atomicOr(stage + k + 2, top);
            };
            if (n_d == 0) {
                put((uint64_t)(nibbles4(v.x) | nibbles4(v.y) << 16) |
                    (uint64_t)(nv > 8 ? nibbles4(v.z) | nibbles4(v.w) << 16 : 0u) << 32);
            } else {
                const uint32_t words[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (uint32_t q = 0; q < 4; ++q) {
                    uint64_t n = 0;
                    uint32_t len = 0;
#pragma unroll
                    for (uint32_t k = 0; k < 4; ++k) {
                        const uint32_t op = (words[q] >> (8 * k)) & 0xFFu, c = op & 7u;
                        if (4 * q + k < nv) {
                            n |= (uint64_t)((c << 1) | ((op >> 3) & 1u)) << (4 * len++);
                            if (c == OP_PD) n |= (uint64_t)(op >> 4) << (4 * len++);
                        }
                    }
                    put(n);
                    s += len;
                }
            }
            __syncthreads();
            pos += total & 0xFFFFu;
            pa += total >> 16;
            // whole chunks leave; what is left of the last one moves to the front
            const uint32_t full = (pos - base) / 32;
            for (uint32_t q = tid; q < full; q += T) chunk_out(q);
            const uint32_t rest = tid < 4 ? stage[4 * full + tid] : 0u;
            __syncthreads();
            for (uint32_t k = tid; k < 4 * full + 4; k += T) stage[k] = k < 4 ? rest : 0u;
            base += 32 * full;
        }
        __syncthreads();
        if (tid == 0 && pos > base) chunk_out(0);
        if (ok)
            for (uint32_t k = tid; k < P; k += T) A.pal_pool[pal_off + k] = k ? B.pal_lab[k - 1] : root;
        __syncthreads();
        if (sample && tid < 16 && S.hist[tid]) atomicAdd(A.misc + 2 + tid, (unsigned long long)S.hist[tid]);
        if (tid == 0) {
            EncMeta m;
            m.nib_off = nib_off;
            m.pal_off = pal_off;
            m.enc_off = S.enc_off;
            m.P = P;
            m.nsym = nsym;
            m.nbytes = nbytes;
            m.n_ops = n_ops;
            m.id = morton3(bx + A.bx0, by, bz);
            m.flags = (root_const ? EF_UNIFORM : 0u) | (ok ? 0u : EF_OVERFLOW);
            m.n_ck = n_ck;
            m.E = 0;
            m.sel = sel;
            m.ck_off = ck_ok ? (uint32_t)ck_off : 0u;
#pragma unroll
            for (uint32_t k = 0; k < 8; ++k) m.level_start[k] = k + 1 < A.L ? 8u * S.level_r[k] : n_ops;
            A.meta[i] = m;
        }
        __syncthreads();
    }
}

// Exhaustive statistics for the mode / table choice: per brick and mode, the
// histogram of the 16 nibble values the rANS coder would see (root nibble, op
// nibbles, Pd offsets and the pad nibble of an odd count).  A mode only changes which
// of several matches an op names: the ops that match nothing, and so the palette, are
// every mode's, and a mode's other nibbles follow from how often each set of matches
// occurs.  So one pass over the children counts the sets (32 with the stop bit, one lane
// each, by ballots) for all modes: 150 bricks of 64^3 19.4 -> 0.25 ms against an op stream
// and a walk per mode.
template <int T, int PER_SM>
__global__ void __launch_bounds__(T, PER_SM) enc_stats_kernel(EncArgs A, uint32_t* __restrict__ hist_out) {
    extern __shared__ __align__(16) uint8_t enc_dyn[];
    __shared__ EncFixed S;
    const uint32_t tid = threadIdx.x, lane = tid & 31, FULL = 0xFFFFFFFFu;
    BrickCtx B = enc_ctx<T>(A, S, enc_dyn);
    uint32_t* sets = S.hist + 16;  // [set << 1 | stop]
    for (;;) {
        if (tid == 0) S.work = atomicAdd(reinterpret_cast<unsigned int*>(A.misc + kMiscQueue), 1u);
        __syncthreads();
        const uint32_t i = S.work;
        if (i >= A.nb) break;
        enc_place(B, i / (A.nbz * A.nby), (i / A.nbz) % A.nby, i % A.nbz);
        const uint32_t n_act = build_pyramid<T>(B), n_ops = 8 * n_act;
        if (tid < 64) S.hist[tid] = 0;
        __syncthreads();
        const uint64_t root = B.lab[0];
        uint32_t count = 0;  // of the set and stop bit numbered as this lane
        for_children<T>(B, true, [&](uint32_t r, uint32_t c, uint32_t set, uint32_t stop, uint64_t label) {
            const uint32_t key = set << 1 | (stop & 1u);
            uint32_t m = __ballot_sync(FULL, stop < 2);
#pragma unroll
            for (uint32_t k = 0; k < 5; ++k) {
                const uint32_t b = __ballot_sync(FULL, (key >> k) & 1u);
                m &= (lane >> k) & 1u ? b : ~b;
            }
            count += __popc(m);
            const bool need = stop < 2 && set == 0;
            const uint32_t needs = __ballot_sync(FULL, need);
            if (stop < 2) {
                if (need) {
                    B.ops[8 * r + c] = (uint8_t)(stop << 3);
                    B.pal_lab[8 * r + c] = label;
                }
                if (c == 0) B.need8[r] = (uint8_t)(needs >> (lane & 24u));
            }
        });
        if (count) atomicAdd(sets + lane, count);
        __syncthreads();
        palette_walk<T>(B, root, n_act, [&](uint32_t j, uint32_t code, uint32_t delta) {
            atomicAdd(&S.hist[code << 1 | (B.ops[j] >> 3 & 1u)], 1u);
            if (code == OP_PD) atomicAdd(&S.hist[delta], 1u);
        });
        if (tid == 0) {
            S.hist[(OP_PA << 1) | (n_act == 0 ? 1u : 0u)] += 1;     // root nibble
            if ((1 + n_ops + S.n_pd) & 1u) S.hist[0] += 1;          // pad nibble
        }
        __syncthreads();
        for (uint32_t k = tid; k < kModes * 16; k += T) {
            const uint32_t mode = k >> 4, nib = k & 15u;
            const uint64_t codes = kModeTable.t[mode];
            uint32_t n = S.hist[nib];
            for (uint32_t set = 1; set < 16; ++set)
                if (((uint32_t)(codes >> (3 * set)) & 7u) == nib >> 1) n += sets[set << 1 | (nib & 1u)];
            hist_out[(size_t)i * kModes * 16 + k] = n;
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------ K2 model
// buildRansModel (brickEncoding.cpp:146-200) plus per-symbol constants for the
// encoder: M = ceil(2^(31+s) / f) with s = ceil(log2 f) gives floor(x / f) =
// (x * M) >> (31 + s) exactly for every x < 2^31 (the encoder's state bound):
// M = 2^(31+s)/f + e with 0 <= e < 1 adds less than x / 2^(31+s) < 2^-s <= 1/f
// to x/f, whose fractional part is at most 1 - 1/f (Granlund & Montgomery 1994).
// One warp, a lane per symbol: 8 -> 3 us against one thread.
__global__ void model_kernel(const unsigned long long* hist, uint32_t* model) {
    const uint32_t i = threadIdx.x, FULL = 0xFFFFFFFFu;
    const bool on = i < 16;
    uint32_t freq = on ? max((uint32_t)hist[i], 1u) : 0u;  // size_t -> uint32_t as :157
    uint64_t raw = freq;
    for (int d = 16; d > 0; d >>= 1) raw += __shfl_xor_sync(FULL, raw, d);
    if (on) freq = (uint32_t)max((uint64_t)freq * kTot / raw, (uint64_t)1);
    uint32_t norm = __reduce_add_sync(FULL, freq);
    if (norm < kTot && i == 0) freq += kTot - norm;
    for (; norm > kTot; --norm) {  // (at most 16 too many) from the first of the largest
        const uint32_t most = __reduce_max_sync(FULL, freq);
        if (most <= 1) break;
        const uint32_t first = __ffs(__ballot_sync(FULL, freq == most)) - 1;
        if (i == first) --freq;
    }
    uint32_t end = freq;
    for (int d = 1; d < 16; d <<= 1) {
        const uint32_t y = __shfl_up_sync(FULL, end, d);
        if ((int)i >= d) end += y;
    }
    if (on) {
        model[i] = freq;
        model[16 + i] = end - freq;
        const uint32_t s = freq > 1 ? 32 - __clz(freq - 1) : 0;
        model[33 + i] = (uint32_t)(((1ull << (31 + s)) + freq - 1) / freq);
        model[49 + i] = 31 + s;
    }
    if (i == 15) model[32] = end;
}

// ------------------------------------------------------------ K3 rANS
// ransEncodeSymbol (brickEncoding.cpp:202-219) on the state x < 2^31 (brickEncoding:
// 2^19 f after renormalisation, times 4096 / f):
//     y = x without the bytes that leave (one when x >= f << 19, a second when
//         x >= f << 27, which takes f < 16)
//     x' = y + start + (y / f) (4096 - f)
// as a chain of steps that put out at most one byte each, all of one form:
//     x' = x >= bound ? (x >> 8) + start + ((h >> s) >> 8) mul : x + start + (h >> s) mul,
//     h = the high half of x M
// With M = ceil(2^(31 + ceil(log2 f)) / f), h >> s is exactly x / f (Granlund &
// Montgomery, as model_kernel), and (x >> 8) / f is (x / f) >> 8, so both outcomes come
// from one multiplication and the comparison is off the chain of multiply, shift,
// multiply-add, select: 23 cycles (measured; 38 with the select first, whose comparison
// alone takes about 14).  A symbol with f < 16 takes a step before that only drops a
// byte (M = mul = 0); f = 1, which has no such M, takes two, then M = 2^32 - 1, which
// gives x - 1, and start + 4095.  An entry is {M, bound, mul, start << 5 | s}.
__device__ __forceinline__ uint4 rans_entry(const uint32_t* __restrict__ md, uint32_t s) {
    const uint32_t f = md[s], start = md[16 + s], sh = md[49 + s] - 31;
    return f == 1 ? make_uint4(0xFFFFFFFFu, 0xFFFFFFFFu, kTot - f, (start + kTot - 1) << 5)
                  : make_uint4(md[33 + s], f << 19, kTot - f, start << 5 | (sh - 1));
}
__device__ __forceinline__ void rans_enc_step(uint32_t& x, const uint4 t) {
    const uint32_t h = __umulhi(x, t.x), start = t.w >> 5;
    const uint32_t xa = x + start + __funnelshift_r(h, 0u, t.w) * t.z;  // (shifts by t.w & 31)
    const uint32_t xb = (x >> 8) + start + __funnelshift_r(h, 0u, t.w + 8) * t.z;
    x = x >= t.y ? xb : xa;
}

// A brick's symbols are one dependent chain, and the longest brick's is the kernel's
// time, so one warp of a block does nothing else: lane k runs brick k's steps, in
// batches of 64 or 256, on entries read ahead from shared memory, and leaves the states
// there.  Each of the K bricks has a warp of its own that meanwhile turns the next
// symbols into steps and works out from the last batch's states the bytes they put out,
// their place (a ballot prefix) and the seek checkpoints among them; its global loads
// come 1024 symbols (nibbles) or 32 checkpoints at a time.  K = 1 while there are no
// more bricks than warp schedulers, so that no chain shares one; beyond, several chains
// per warp, since a chain's step costs the scheduler as much for one lane as for many.
// Measured against one lane per brick that did all of it (165 cycles per symbol): 512
// bricks of 64^3, longest 84,720 symbols, 7.24 -> 1.24 ms (K = 1, 28 cycles per
// symbol); 8192 bricks of 32^3 0.91 -> 0.30 ms (K = 8; 0.67 with K = 1); 60 bricks of
// 32^3 0.60 -> 0.11 ms.  Batches of 128 with K = 1: 1.28 ms, of 512: 1.22
// ms, but 60 bricks of 32^3 take 0.113 ms for 0.105.
template <uint32_t kRansBatch>
struct RansBrick {
    static constexpr uint32_t kRing = 4 * kRansBatch;
    uint4 ring[kRing];          // steps, in order, modulo kRing
    uint4 tab[16];              // the model's entries
    uint4 nib[32];              // packed nibbles of 1024 symbols
    uint32_t x[2][kRansBatch];  // the state before each step of two batches
    uint32_t end[2];            // and after their last one
    uint16_t ck[kRing];         // 1 + the checkpoint whose symbol the step completes, or 0
};
static_assert(sizeof(RansBrick<64>) % 128 == 16, "eight bricks' entries are read from different banks");
template <int K, uint32_t kRansBatch>
__global__ void __launch_bounds__(32 * (K + 1)) enc_rans_kernel(EncMeta* __restrict__ meta, uint32_t nb,
                                                                const uint8_t* __restrict__ nib_pool,
                                                                uint64_t* __restrict__ rec_size, uint32_t rec_fixed,
                                                                uint8_t* __restrict__ enc_pool,
                                                                const uint32_t* __restrict__ model, uint32_t n_tables,
                                                                Checkpoint* __restrict__ ck_all) {
    constexpr uint32_t kRansRing = RansBrick<kRansBatch>::kRing;
    __shared__ RansBrick<kRansBatch> s_bricks[K];
    const uint32_t lane = threadIdx.x & 31, FULL = 0xFFFFFFFFu;
    // The chain's warp.  Warps take an SM's four schedulers in turn, by slot; of blocks of two warps, the first
    // pair of blocks has its chains in their first warps and the next one in their second, so that four chains do
    // not meet (512 bricks of 64^3 1.47 -> 1.28 ms against every other block).  Five and nine warps differ by one.
    const uint32_t warp = threadIdx.x >> 5;
    uint32_t chain_warp = 0;
    if (K == 1) {
        __shared__ uint32_t s_slot;
        if (threadIdx.x == 0) asm volatile("mov.u32 %0, %%warpid;" : "=r"(s_slot));
        __syncthreads();
        chain_warp = s_slot >> 2 & 1u;
    }
    if (warp == chain_warp) {
        auto& B = s_bricks[min(lane, (uint32_t)K - 1)];
        uint32_t x = kRansL;
        uint4 ea[8], eb[8];
        auto fetch = [&](const uint4* r, uint4 (&e)[8]) {
#pragma unroll
            for (int k = 0; k < 8; ++k) e[k] = r[k];
        };
        auto code = [&](const uint4 (&e)[8], uint4* xs) {
            uint32_t st[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                st[k] = x;
                rans_enc_step(x, e[k]);
            }
            xs[0] = make_uint4(st[0], st[1], st[2], st[3]);
            xs[1] = make_uint4(st[4], st[5], st[6], st[7]);
        };
        __syncthreads();
        for (uint32_t n = 0;; ++n) {
            if (lane < K) {
                const uint4* ring = B.ring + (n * kRansBatch) % kRansRing;
                uint4* xs = reinterpret_cast<uint4*>(B.x[n & 1]);
                fetch(ring, ea);
#pragma unroll 1
                for (uint32_t k = 0; k < kRansBatch / 16; ++k) {
                    fetch(ring + 8, eb);
                    code(ea, xs);
                    ring += 16;
                    if (k + 1 < kRansBatch / 16) fetch(ring, ea);
                    code(eb, xs + 2);
                    xs += 4;
                }
                B.end[n & 1] = x;
            }
            if (!__syncthreads_or(0)) return;
        }
    }
    const uint32_t kb = chain_warp ? warp : warp - 1, i = blockIdx.x * K + kb;
    auto& B = s_bricks[kb];
    uint32_t n_sym = 0, n_ck = 0, tables = 0;
    uint64_t nib_off = 0;
    Checkpoint* ck = ck_all;
    uint8_t* out = enc_pool;
    const bool have = i < nb && !(meta[i].flags & EF_OVERFLOW);
    if (have) {
        const EncMeta& m = meta[i];
        n_sym = 2 * m.nbytes;  // symbols coded, the pad nibble of an odd count included
        n_ck = m.n_ck;
        nib_off = m.nib_off;
        tables = min((m.sel >> 4) & 15u, n_tables - 1);
        ck += m.ck_off;
        out += m.enc_off;
    }
    if (lane < 16) B.tab[lane] = rans_entry(model + tables * kModelWords, lane);
    // the packed nibbles start 16-byte aligned and are padded to 16: a chunk of 32 symbols is 16 bytes
    const uint4* src = reinterpret_cast<const uint4*>(nib_pool + nib_off);
    const uint32_t n16 = (n_sym + 31) / 32;
    auto load_nib = [&](int blk) -> uint4 {
        const uint32_t q = 32u * (uint32_t)blk + lane;
        return blk >= 0 && q < n16 ? src[q] : make_uint4(0, 0, 0, 0);
    };
    // checkpoints (they have ascending symbols; the chain runs backwards): lane l holds the symbol of
    // checkpoint ck_base - 1 - l; n_ck are left.  A chunk has at most two (16 ops apart).
    uint32_t ck_base = n_ck, ck_sym = lane < n_ck ? ck[n_ck - 1 - lane].sym : 0u;
    const uint32_t lt = (1u << lane) - 1u, le = (2u << lane) - 1u;
    int chunk = (int)n16 - 1;  // the next chunk to turn into steps
    uint4 nib_next = load_nib(chunk >> 5);
    bool fresh = true;         // nib_next is the chunk's block
    uint32_t made = 0;         // steps so far
    uint32_t n_batches = have ? 0xFFFFFFFFu : 0u;  // known once every symbol has its steps
    const uint32_t rel = 31 - lane;  // lane l takes the chunk's symbol 31 - l (a byte's low nibble is the later one)
    auto produce = [&](uint32_t target) {
        while (made < target && chunk >= 0) {
            if (fresh || (chunk & 31) == 31) {
                __syncwarp();
                B.nib[lane] = nib_next;
                nib_next = load_nib((chunk >> 5) - 1);
                fresh = false;
                __syncwarp();
            }
            const uint32_t sym = 32u * (uint32_t)chunk + rel;
            const uint32_t byte = reinterpret_cast<const uint8_t*>(B.nib)[16 * (chunk & 31) + (rel >> 1)];
            const uint4 t = B.tab[(rel & 1u) ? byte & 15u : byte >> 4];
            const bool valid = sym < n_sym;
            const bool one = t.x == 0xFFFFFFFFu, few = one || t.y < (16u << 19);  // f = 1, f < 16
            const uint32_t m0 = __ballot_sync(FULL, valid), m1 = __ballot_sync(FULL, valid && few),
                           m2 = __ballot_sync(FULL, valid && one);
            // the chunk's checkpoints, as a mask of its steps' order
            const uint32_t due = lane >= ck_base - n_ck && lane < ck_base && (ck_sym >> 5) == (uint32_t)chunk
                                     ? 0x80000000u >> (ck_sym & 31u)
                                     : 0u;
            const uint32_t mc = __reduce_or_sync(FULL, due);
            if (valid) {
                uint32_t s = made + __popc(m0 & lt) + __popc(m1 & lt) + __popc(m2 & lt);
                if (few) {
                    const uint32_t f = one ? 1u : t.y >> 19;
                    B.ring[s % kRansRing] = make_uint4(0u, f << 27, 0u, 0u);
                    B.ck[s % kRansRing] = 0;
                    ++s;
                }
                if (one) {
                    B.ring[s % kRansRing] = make_uint4(0u, 1u << 19, 0u, 0u);
                    B.ck[s % kRansRing] = 0;
                    ++s;
                }
                B.ring[s % kRansRing] = t;
                B.ck[s % kRansRing] = (mc >> lane) & 1u ? (uint16_t)(n_ck - __popc(mc & lt)) : (uint16_t)0;
            }
            made += __popc(m0) + __popc(m1) + __popc(m2);
            n_ck -= __popc(mc);
            if (ck_base - n_ck > 30 && n_ck) {
                ck_base = n_ck;
                ck_sym = lane < n_ck ? ck[n_ck - 1 - lane].sym : 0u;
            }
            --chunk;
        }
        if (chunk < 0 && n_batches == 0xFFFFFFFFu) {  // the last batch is filled up with steps that do nothing
            n_batches = (made + kRansBatch - 1) / kRansBatch;
            for (uint32_t s = made + lane; s < n_batches * kRansBatch; s += 32) {
                B.ring[s % kRansRing] = make_uint4(0u, 0xFFFFFFFFu, 0u, 0u);
                B.ck[s % kRansRing] = 0;
            }
        }
    };
    if (have) produce(kRansBatch);
    uint32_t emitted = 0;
    __syncthreads();
    for (uint32_t n = 0;; ++n) {
        if (n >= 1 && n <= n_batches) {  // what batch n - 1 put out
            const uint32_t d = (n - 1) & 1u;
#pragma unroll
            for (uint32_t h = 0; h < kRansBatch / 32; ++h) {
                const uint32_t j = 32 * h + lane, s = ((n - 1) * kRansBatch + j) % kRansRing;
                const uint32_t x = B.x[d][j], id = B.ck[s];
                const uint32_t b = __ballot_sync(FULL, x >= B.ring[s].y);
                if ((b >> lane) & 1u) out[emitted + __popc(b & lt)] = (uint8_t)x;
                if (id) {  // a checkpoint's state, the decoder's before its symbol, is the encoder's after it
                    ck[id - 1].state = j + 1 < kRansBatch ? B.x[d][j + 1] : B.end[d];
                    ck[id - 1].pos = emitted + __popc(b & le);
                }
                emitted += __popc(b);
            }
            if (n == n_batches) {
                const uint32_t x = B.end[d];
                if (lane < 4) out[emitted + lane] = (uint8_t)(x >> (8 * lane));  // ransFlush, little-endian
                if (lane == 0) {
                    meta[i].E = emitted + 4;
                    rec_size[i] = rec_fixed + 8ull * meta[i].P + emitted + 4;  // the brick's record in the image
                }
            }
            __syncwarp();  // its steps make room for new ones
        }
        if (n_batches == 0xFFFFFFFFu) produce((n + 2) * kRansBatch);
        if (!__syncthreads_or(n < n_batches)) return;
    }
}

// ------------------------------------------------------------ K4 serialize
// The records' sizes become their places in the image, after a header of `first` bytes;
// the image's length goes to *total.  One block, 4096 records a turn.
__global__ void __launch_bounds__(1024) place_kernel(uint64_t* __restrict__ rec, uint32_t nb, uint64_t first,
                                                     unsigned long long* __restrict__ total) {
    __shared__ uint64_t sh[33];
    for (uint32_t base = 0; base < nb; base += 4096) {
        const uint32_t i = base + 4 * threadIdx.x;
        uint64_t v[4], sum = 0, all;
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) sum += v[k] = i + k < nb ? rec[i + k] : 0ull;
        uint64_t at = first + block_exclusive<uint64_t>(sum, sh, &all);
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) {
            if (i + k < nb) rec[i + k] = at;
            at += v[k];
        }
        first += all;
    }
    if (threadIdx.x == 0) *total = first;
}

// `n` bytes from src to dst by the block, whole words of dst where they can be (from two words
// of src): 6.5 MB of 512 bricks' records 47 -> 13 us, 4.8 MB of 320 bricks' 65 -> 17 us against a
// byte per thread.
__device__ __forceinline__ void copy_bytes(uint8_t* __restrict__ dst, const uint8_t* __restrict__ src, uint64_t n) {
    const uint64_t head = min(n, (uint64_t)(-(uintptr_t)dst & 3u)), words = (n - head) / 4, tail = head + 4 * words;
    const uint32_t* w = reinterpret_cast<const uint32_t*>((uintptr_t)(src + head) & ~(uintptr_t)3);
    const uint32_t sh = 8 * ((uintptr_t)(src + head) & 3u);
    for (uint64_t k = threadIdx.x; k < words; k += blockDim.x)
        reinterpret_cast<uint32_t*>(dst + head)[k] = __funnelshift_r(w[k], sh ? w[k + 1] : 0u, sh);
    if (threadIdx.x < head) dst[threadIdx.x] = src[threadIdx.x];
    if (threadIdx.x < n - tail) dst[tail + threadIdx.x] = src[tail + threadIdx.x];
}

// One block per brick record: ID, P, palette, E, stream, nSymbols (fileIO.cpp:57-96).
// Version 2 adds a u32 after the ID: the brick's table (bits 4..7) and mode (bits 0..3).
// Block nb writes the header: version 1, 152 bytes (fileIO.cpp:25-49); version 2, 28 bytes
// and 128 per table.  Nothing is written when the image is longer than `cap`.
__global__ void serialize_kernel(const EncMeta* __restrict__ meta, uint32_t nb, const uint64_t* __restrict__ rec_off,
                                 const uint64_t* __restrict__ pal_pool, const uint8_t* __restrict__ enc_pool,
                                 uint8_t* __restrict__ image, uint64_t cap, const unsigned long long* __restrict__ len,
                                 const uint32_t* __restrict__ model, uint32_t n_tables, uint32_t b) {
    if (*len > cap) return;
    const uint32_t i = blockIdx.x;
    const bool v2 = n_tables > 0;
    if (i == nb) {
        uint32_t* hdr = reinterpret_cast<uint32_t*>(image);
        // the reference always writes BRICK_SIZE after the brick count (fileIO.cpp:28)
        const uint32_t fixed[7] = {kMagic, v2 ? 2u : 1u, nb, b, 16u, model[32], n_tables};
        if (threadIdx.x == 0)
            for (uint32_t k = 0; k < (v2 ? 7u : 6u); ++k) hdr[k] = fixed[k];
        for (uint32_t k = threadIdx.x; k < 32 * max(1u, n_tables); k += blockDim.x)
            hdr[(v2 ? 7 : 6) + k] = model[(k >> 5) * kModelWords + (k & 31u)];
        return;
    }
    const EncMeta m = meta[i];
    uint8_t* dst = image + rec_off[i];
    const uint8_t* pal = reinterpret_cast<const uint8_t*>(pal_pool + m.pal_off);
    const uint8_t* enc = enc_pool + m.enc_off;
    const uint32_t h = v2 ? 12 : 8;  // ID [, sel], P
    if (threadIdx.x < h + 8) {
        const uint32_t k = threadIdx.x;
        const uint32_t word = k < 4 ? m.id : k < h - 4 ? m.sel & 0xFFu : k < h ? m.P : k < h + 4 ? m.E : m.nsym;
        const uint64_t at = k < h ? k : k < h + 4 ? k + 8ull * m.P : k + 8ull * m.P + m.E;
        dst[at] = (uint8_t)(word >> (8 * (k & 3u)));
    }
    copy_bytes(dst + h, pal, 8ull * m.P);
    copy_bytes(dst + h + 4 + 8ull * m.P, enc, m.E);
}

// ------------------------------------------------------------ host driver
namespace {

template <class T>
cudaError_t grow(T** p, size_t* cap, size_t need) {
    if (*p && *cap >= need) return cudaSuccess;
    cudaFree(*p);
    *p = nullptr;
    *cap = 0;
    size_t n = std::max<size_t>(need, 1);
    cudaError_t e = cudaMalloc(p, n * sizeof(T));
    if (e == cudaSuccess) *cap = n;
    return e;
}

int sm_count(int device) {
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    return std::max(1, sms);
}

// K1's two forms.  64^3 bricks: one CTA of 1024 threads per SM (512 bricks 0.76 ms, 150
// bricks 0.26 ms; 384 threads, four per SM: 0.85 and 0.42 ms -- a brick in flight takes
// 2 MB of the L2 that its second look at the voxels wants to find them in).  Smaller
// bricks, whose phases are short against their barriers: 320 threads, four per SM (8192
// bricks of 32^3 0.66 ms, against 1.27 ms); 32^3 ones no more than there are SMs take
// the first form (60 bricks 54 against 69 us).
bool enc_wide(uint32_t L, uint32_t nb, int device) { return L >= 7 || (L == 6 && nb <= (uint32_t)sm_count(device)); }
template <class F>
auto enc_form(bool wide, F f) {
    return wide ? f(std::integral_constant<int, 1024>(), std::integral_constant<int, 1>())
                : f(std::integral_constant<int, 320>(), std::integral_constant<int, 4>());
}

size_t enc_scratch_per_cta(uint32_t L, bool wide) {
    return enc_form(wide, [&](auto t, auto) -> size_t { return enc_scratch<decltype(t)::value>(L).bytes; });
}

// CTAs of K1 or the statistics kernel that the device holds.
int g_enc_occ[64][8][2] = {};
uint32_t enc_grid(int device, uint32_t L, bool wide) {
    int& occ = g_enc_occ[device & 63][L & 7][wide];
    if (occ == 0)
        occ = enc_form(wide, [&](auto t, auto n) {
            constexpr int T = decltype(t)::value, N = decltype(n)::value;
            int a = 0, b = 0;
            for (const void* k : {(const void*)enc_bricks_kernel<T, N>, (const void*)enc_stats_kernel<T, N>})
                cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)enc_smem<T>(7));
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, enc_bricks_kernel<T, N>, T, enc_smem<T>(L));
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, enc_stats_kernel<T, N>, T, enc_smem<T>(L));
            return std::max(1, std::min(a, b)) * sm_count(device);
        });
    return (uint32_t)occ;
}

}  // namespace

// Runs K1..K4 on a device volume; leaves the image in s->d_image.
// buildRansModel's per-symbol encoder constants for a given normalised table
// (the host side of model_kernel).
void table_model(const uint32_t* freq, uint32_t* model) {
    uint32_t acc = 0;
    for (int i = 0; i < 16; ++i) {
        model[i] = freq[i];
        model[16 + i] = acc;
        acc += freq[i];
        uint32_t s = 0;
        while ((1u << s) < freq[i]) ++s;
        const uint64_t M = ((1ull << (31 + s)) + freq[i] - 1) / freq[i];
        model[33 + i] = (uint32_t)M;
        model[49 + i] = 31 + s;
    }
    model[32] = acc;
}

int check_tables(const EncodeSelection* sel, std::string& err) {
    if (!sel || sel->n_tables == 0) return CSV_OK;
    if (sel->n_tables > kMaxTables) {
        err = "at most 16 shared rANS tables";
        return CSV_ERANGE;
    }
    for (uint32_t t = 0; t < sel->n_tables; ++t) {
        uint32_t sum = 0;
        for (int k = 0; k < 16; ++k) {
            if (sel->freq[t][k] == 0) {
                err = "a table frequency is 0";
                return CSV_EINVAL;
            }
            sum += sel->freq[t][k];
        }
        if (sum != kTot) {
            err = "a table's frequencies do not sum to 4096";
            return CSV_EINVAL;
        }
    }
    return CSV_OK;
}

// Per brick and mode, the 16-bin nibble histogram (the exhaustive search's statistics).
int encode_stats(EncoderState* s, int device, const uint64_t* d_vol, uint64_t W, uint64_t H, uint64_t D, uint32_t b,
                 uint32_t* d_hist, cudaStream_t st, std::string& err) {
    const uint64_t nbx = (W + b - 1) / b, nby = (H + b - 1) / b, nbz = (D + b - 1) / b;
    if (nbx > 1024 || nby > 1024 || nbz > 1024) {
        err = "volume needs more than 1024 bricks along an axis";
        return CSV_ERANGE;
    }
    const uint32_t nb = (uint32_t)(nbx * nby * nbz);
    cudaError_t e;
    if (!s->d_misc && (e = cudaMalloc(&s->d_misc, kMiscWords * sizeof(unsigned long long))) != cudaSuccess) {
        err = cudaGetErrorString(e);
        return CSV_ECUDA;
    }
    const bool wide = enc_wide(levels_of(b), nb, device);
    const uint32_t grid = std::min<uint32_t>(enc_grid(device, levels_of(b), wide), std::max<uint32_t>(nb, 1));
    const size_t per_cta = enc_scratch_per_cta(levels_of(b), wide);
    if ((e = grow(&s->d_scratch, &s->scratch_cap, per_cta * grid)) != cudaSuccess ||
        (e = cudaMemsetAsync(s->d_misc, 0, kMiscWords * sizeof(unsigned long long), st)) != cudaSuccess) {
        err = cudaGetErrorString(e);
        return CSV_ECUDA;
    }
    EncArgs A;
    memset(&A, 0, sizeof A);
    A.vol = d_vol;
    A.W = W; A.H = H; A.D = D;
    A.b = b; A.L = levels_of(b);
    A.nbx = (uint32_t)nbx; A.nby = (uint32_t)nby; A.nbz = (uint32_t)nbz;
    A.nb = nb;
    A.scratch = s->d_scratch;
    A.scratch_per_cta = per_cta;
    A.misc = s->d_misc;
    A.pairs = W % 2 == 0 && (uintptr_t)d_vol % 16 == 0;
    if (nb)
        enc_form(wide, [&](auto t, auto n) {
            constexpr int T = decltype(t)::value;
            enc_stats_kernel<T, decltype(n)::value><<<grid, T, enc_smem<T>(A.L), st>>>(A, d_hist);
            return 0;
        });
    if ((e = cudaGetLastError()) != cudaSuccess) {
        err = cudaGetErrorString(e);
        return CSV_ECUDA;
    }
    return CSV_OK;
}

#define CK(x)                                                              \
    do {                                                                   \
        if ((e = (x)) != cudaSuccess) {                                    \
            err = std::string(#x) + ": " + cudaGetErrorString(e);          \
            return CSV_ECUDA;                                              \
        }                                                                  \
    } while (0)

// K3 + K4 (and the model) after K1: the model from the sample histogram in
// misc[2..17] (or the selection's tables), then the rANS pass and the image.
static int finish_encode(EncoderState* s, const EncodeSelection* sel, cudaStream_t st, std::string& err);

int encode_device(EncoderState* s, int device, const uint64_t* d_vol, uint64_t W, uint64_t H, uint64_t D, uint32_t b,
                  cudaStream_t st, std::string& err, const EncodeSelection* sel, const EncodeShard* shard,
                  uint64_t* hist_out) {
    s->valid = false;
    s->device = device;
    s->b = b;
    s->L = levels_of(b);
    s->W = W; s->H = H; s->D = D;
    const uint64_t nbx = (W + b - 1) / b, nby = (H + b - 1) / b, nbz = (D + b - 1) / b;
    const uint64_t nb64 = nbx * nby * nbz;
    if (nbx > 1024 || nby > 1024 || nbz > 1024 || nb64 > 0xFFFFFFFFull) {
        err = "volume needs more than 1024 bricks along an axis (10-bit Morton brick IDs, utils.cpp:10-14)";
        return CSV_ERANGE;
    }
    const uint32_t nb = (uint32_t)nb64;
    s->nb = nb;
    const uint64_t nvox = W * H * D;
    cudaError_t e;
    {
        int rc = check_tables(sel, err);
        if (rc) return rc;
    }
    if (hist_out && sel && sel->n_tables) {
        err = "a shard encodes version-1 images only";
        return CSV_EINVAL;
    }
    s->bricks_done = false;
    CK(grow(&s->d_meta, &s->meta_cap, nb));
    if (!s->d_model) CK(cudaMalloc(&s->d_model, kMaxTables * kModelWords * sizeof(uint32_t)));
    {
        static_assert(sizeof(unsigned long long) == 8, "");
        if (!s->d_misc) CK(cudaMalloc(&s->d_misc, kMiscWords * sizeof(unsigned long long)));
    }
    if (!s->h_words) CK(cudaMallocHost(&s->h_words, sizeof *s->h_words));
    const bool wide = enc_wide(levels_of(b), nb, device);
    const uint32_t grid = std::min<uint32_t>(enc_grid(device, levels_of(b), wide), std::max<uint32_t>(nb, 1));
    const size_t per_cta = enc_scratch_per_cta(levels_of(b), wide);
    CK(grow(&s->d_scratch, &s->scratch_cap, per_cta * grid));
    size_t nib_need = std::max<size_t>(1 << 20, nvox / 4 + 16ull * nb);
    size_t pal_need = std::max<size_t>(1 << 16, nvox / 256 + 64ull * nb);
    // as many ops as the nibble estimate allows (a nibble or two each)
    size_t ck_need = std::max<size_t>(1 << 12, nib_need * 2 / s->S + nb);
    for (int attempt = 0; attempt < 2; ++attempt) {
        if (ck_need > 0xFFFFFFFFull) {  // checkpoint offsets are 32-bit
            err = "volume needs more than 2^32 seek checkpoints";
            return CSV_ERANGE;
        }
        CK(grow(&s->d_nib, &s->nib_cap, nib_need));
        CK(grow(&s->d_pal, &s->pal_cap, pal_need));
        CK(grow(&s->d_ck, &s->ck_cap_total, ck_need));
        CK(cudaMemsetAsync(s->d_misc, 0, kMiscWords * sizeof(unsigned long long), st));
        EncArgs A;
        A.vol = d_vol;
        A.W = W; A.H = H; A.D = D;
        A.b = b; A.L = s->L;
        A.nbx = (uint32_t)nbx; A.nby = (uint32_t)nby; A.nbz = (uint32_t)nbz;
        A.nb = nb;
        A.scratch = s->d_scratch;
        A.scratch_per_cta = per_cta;
        A.meta = s->d_meta;
        A.nib_pool = s->d_nib;
        A.nib_cap = s->nib_cap;
        A.pal_pool = s->d_pal;
        A.pal_cap = s->pal_cap;
        A.ck = s->d_ck;
        A.ck_cap = s->ck_cap_total;
        A.misc = s->d_misc;
        A.sel = sel ? sel->d_sel : nullptr;
        A.bx0 = shard ? shard->bx0 : 0u;
        A.index_base = shard ? shard->index_base : 0u;
        A.pairs = W % 2 == 0 && (uintptr_t)d_vol % 16 == 0;
        if (nb > 0) {
            enc_form(wide, [&](auto t, auto n) {
                constexpr int T = decltype(t)::value;
                enc_bricks_kernel<T, decltype(n)::value><<<grid, T, enc_smem<T>(A.L), st>>>(A);
                return 0;
            });
            CK(cudaGetLastError());
        }
        const unsigned long long* misc = s->h_words->misc;
        CK(cudaMemcpyAsync(s->h_words->misc, s->d_misc, sizeof s->h_words->misc, cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        s->ck_used = misc[kMiscCk];
        s->enc_need = misc[kMiscEnc];
        if (misc[0] <= s->nib_cap && misc[1] <= s->pal_cap && misc[kMiscCk] <= s->ck_cap_total) break;
        if (attempt == 1) {
            err = "encoder pools overflowed twice";
            return CSV_ENOMEM;
        }
        nib_need = std::max<size_t>(nib_need, misc[0]);
        pal_need = std::max<size_t>(pal_need, misc[1]);
        ck_need = std::max<size_t>(ck_need, misc[kMiscCk]);
    }
    if (hist_out) {  // a shard: stop here with the sample histogram; finish_encode_shard completes it
        for (int k = 0; k < 16; ++k) hist_out[k] = s->h_words->misc[2 + k];
        s->bricks_done = true;
        return CSV_OK;
    }
    return finish_encode(s, sel, st, err);
}

int finish_encode_shard(EncoderState* s, const uint64_t hist[16], cudaStream_t st, std::string& err) {
    if (!s || !s->bricks_done) {
        err = "no encoder shard waiting for its model on this context";
        return CSV_EINVAL;
    }
    cudaError_t e;
    unsigned long long h[16];
    for (int k = 0; k < 16; ++k) h[k] = hist[k];
    CK(cudaMemcpyAsync(s->d_misc + 2, h, sizeof h, cudaMemcpyHostToDevice, st));
    s->bricks_done = false;
    return finish_encode(s, nullptr, st, err);
}

static int finish_encode(EncoderState* s, const EncodeSelection* sel, cudaStream_t st, std::string& err) {
    cudaError_t e;
    const uint32_t nb = s->nb, b = s->b;
    const uint32_t n_tables = sel ? sel->n_tables : 0;
    const bool v2 = n_tables > 0;
    std::vector<uint32_t> models(kMaxTables * kModelWords, 0);
    if (v2) {  // the caller's shared tables
        for (uint32_t t = 0; t < n_tables; ++t) table_model(sel->freq[t], &models[t * kModelWords]);
        CK(cudaMemcpyAsync(s->d_model, models.data(), n_tables * kModelWords * sizeof(uint32_t),
                           cudaMemcpyHostToDevice, st));
    } else {  // one model from the sampled bricks' histogram (brickEncoding.hpp:481-482)
        model_kernel<<<1, 32, 0, st>>>(s->d_misc + 2, s->d_model);
        CK(cudaGetLastError());
    }
    if (nb > s->h_meta_cap) {
        cudaFreeHost(s->h_meta);
        s->h_meta = nullptr;
        s->h_meta_cap = 0;
        const size_t cap = std::max<size_t>(4096, nb + nb / 2);
        CK(cudaMallocHost(&s->h_meta, sizeof(EncMeta) * cap));
        s->h_meta_cap = cap;
    }
    s->n_tables = std::max<uint32_t>(1, n_tables);
    s->v2 = v2;
    CK(grow(&s->d_enc, &s->enc_cap, std::max<uint64_t>(s->enc_need, 16)));
    CK(grow(&s->d_rec_off, &s->rec_cap, std::max<uint32_t>(nb, 1)));
    if (nb) {
        const uint32_t n_sm = (uint32_t)sm_count(s->device);
        auto rans = [&](auto kernel, uint32_t K) {
            kernel<<<(nb + K - 1) / K, 32 * (K + 1), 0, st>>>(s->d_meta, nb, s->d_nib, s->d_rec_off, v2 ? 20u : 16u,
                                                             s->d_enc, s->d_model, s->n_tables, s->d_ck);
        };
        if (nb <= 4 * n_sm) rans(enc_rans_kernel<1, 256>, 1);
        else if (nb <= 16 * n_sm) rans(enc_rans_kernel<4, 64>, 4);
        else rans(enc_rans_kernel<8, 64>, 8);
        CK(cudaGetLastError());
    }
    place_kernel<<<1, 1024, 0, st>>>(s->d_rec_off, nb, v2 ? 28 + 128ull * n_tables : kHeaderBytes,
                                     s->d_misc + kMiscImage);
    // The image is written without waiting for its length: once more when it is longer than the last one's buffer.
    for (int pass = 0; pass < 2; ++pass) {
        serialize_kernel<<<nb + 1, 256, 0, st>>>(s->d_meta, nb, s->d_rec_off, s->d_pal, s->d_enc, s->d_image, s->image_cap,
                                                 s->d_misc + kMiscImage, s->d_model, n_tables, b);
        CK(cudaGetLastError());
        if (pass == 0) {
            if (nb) CK(cudaMemcpyAsync(s->h_meta, s->d_meta, sizeof(EncMeta) * nb, cudaMemcpyDeviceToHost, st));
            CK(cudaMemcpyAsync(s->h_words->misc + kMiscImage, s->d_misc + kMiscImage, sizeof(unsigned long long),
                               cudaMemcpyDeviceToHost, st));
            if (!v2)
                CK(cudaMemcpyAsync(s->h_words->model, s->d_model, sizeof s->h_words->model, cudaMemcpyDeviceToHost, st));
        }
        CK(cudaStreamSynchronize(st));
        if (s->h_words->misc[kMiscImage] <= s->image_cap) break;
        const uint64_t len = s->h_words->misc[kMiscImage];
        // (the next one may be a little longer; where memory is short, no more than this one takes)
        if (grow(&s->d_image, &s->image_cap, len + len / 8) != cudaSuccess) {
            cudaGetLastError();
            CK(grow(&s->d_image, &s->image_cap, len));
        }
    }
    if (!v2) memcpy(models.data(), s->h_words->model, sizeof s->h_words->model);
    const uint32_t* model = models.data();
    for (uint32_t t = 0; t < s->n_tables; ++t)
        for (int k = 0; k < 16; ++k) {
            s->tab_freq[t][k] = models[t * kModelWords + k];
            s->tab_cum[t][k] = models[t * kModelWords + 16 + k];
        }
    for (int k = 0; k < 16; ++k) {
        s->freq[k] = model[k];
        s->cum[k] = model[16 + k];
    }
    s->cum[16] = model[32];
#undef CK
    s->image_len = s->h_words->misc[kMiscImage];
    s->valid = true;
    return CSV_OK;
}

// Builds a decoder dataset from the last encode (no seek-index pass needed).
int encoder_to_dataset(EncoderState* s, DeviceDataset& d, std::string& err) {
    if (!s || !s->valid) {
        err = "no encoded image on this context";
        return CSV_EINVAL;
    }
    const uint32_t nb = s->nb;
    d.device = s->device;
    d.nb = nb;
    d.b = s->b;
    d.L = s->L;
    d.S = s->S;
    d.total = kTot;
    memcpy(d.freq, s->freq, sizeof d.freq);
    memcpy(d.cum, s->cum, sizeof d.cum);
    std::vector<BrickDesc> desc(std::max<uint32_t>(nb, 1));
    uint64_t pal_n = 0, enc_n = 0;
    d.h_ids = (uint32_t*)malloc(sizeof(uint32_t) * std::max<uint32_t>(1, nb));
    d.h_cost = (uint32_t*)malloc(sizeof(uint32_t) * std::max<uint32_t>(1, nb));
    for (uint32_t i = 0; i < nb; ++i) {
        const EncMeta& m = s->h_meta[i];
        BrickDesc& bd = desc[i];
        memset(&bd, 0, sizeof bd);
        bd.pal_off = m.pal_off;
        bd.enc_off = m.enc_off;
        bd.P = m.P;
        bd.E = m.E;
        bd.nsym = m.nsym;
        bd.id = m.id;
        bd.ck_off = m.ck_off;
        bd.ck_cap = m.n_ck;
        bd.n_ops = m.n_ops;
        bd.flags = ((m.flags & EF_UNIFORM) ? BF_UNIFORM : 0u) | (s->L << BF_LEVELS_SHIFT) |
                   ((s->v2 ? std::min((m.sel >> 4) & 15u, s->n_tables - 1) : 0u) << BF_MODEL_SHIFT);
        for (int k = 0; k < 8; ++k) bd.level_start[k] = m.level_start[k];
        d.h_ids[i] = m.id;
        d.h_cost[i] = m.nsym;
        pal_n = std::max<uint64_t>(pal_n, m.pal_off + m.P);
        enc_n = std::max<uint64_t>(enc_n, m.enc_off + ((m.E + 15) & ~15u));
        d.stream_bytes += m.E;
        d.palette_entries += m.P;
        d.max_nsym = std::max(d.max_nsym, m.nsym);
        d.max_P = std::max(d.max_P, m.P);
    }
    d.ck_entries = s->ck_used;
    d.enc_pool_bytes = std::max<uint64_t>(16, enc_n);
    d.pal_pool_entries = std::max<uint64_t>(1, pal_n);
    d.n_models = s->n_tables;
    std::vector<uint32_t> lut((size_t)kTot * s->n_tables);
    for (uint32_t t = 0; t < s->n_tables; ++t) build_lut(s->tab_freq[t], s->tab_cum[t], &lut[(size_t)t * kTot]);
    d.fast_models = lut_fast_mask(lut.data(), s->n_tables);
    cudaError_t e;
    if ((e = cudaMalloc(&d.d_bricks, sizeof(BrickDesc) * std::max<uint32_t>(1, nb))) != cudaSuccess ||
        (e = cudaMalloc(&d.d_pal, 8 * std::max<uint64_t>(1, pal_n))) != cudaSuccess ||
        (e = cudaMalloc(&d.d_enc, std::max<uint64_t>(16, enc_n))) != cudaSuccess ||
        (e = cudaMalloc(&d.d_ck, sizeof(Checkpoint) * std::max<uint64_t>(1, d.ck_entries))) != cudaSuccess ||
        (e = cudaMalloc(&d.d_lut, sizeof(uint32_t) * lut.size())) != cudaSuccess) {
        err = std::string("device allocation: ") + cudaGetErrorString(e);
        return CSV_ENOMEM;
    }
    if ((e = cudaMemcpy(d.d_bricks, desc.data(), sizeof(BrickDesc) * nb, cudaMemcpyHostToDevice)) != cudaSuccess ||
        (e = cudaMemcpy(d.d_pal, s->d_pal, 8 * pal_n, cudaMemcpyDeviceToDevice)) != cudaSuccess ||
        (e = cudaMemcpy(d.d_enc, s->d_enc, enc_n, cudaMemcpyDeviceToDevice)) != cudaSuccess ||
        (e = cudaMemcpy(d.d_ck, s->d_ck, sizeof(Checkpoint) * d.ck_entries, cudaMemcpyDeviceToDevice)) !=
            cudaSuccess ||
        (e = cudaMemcpy(d.d_lut, lut.data(), sizeof(uint32_t) * lut.size(), cudaMemcpyHostToDevice)) !=
            cudaSuccess) {
        err = std::string("dataset copy: ") + cudaGetErrorString(e);
        return CSV_ECUDA;
    }
    return CSV_OK;
}

const uint8_t* encoder_image(EncoderState* s, size_t* len) {
    if (!s || !s->valid) return nullptr;
    *len = s->image_len;
    return s->d_image;
}

}  // namespace csv
