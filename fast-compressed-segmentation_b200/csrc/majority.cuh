// majority.cuh -- the label of a coarser node (majorityVote8, brick.hpp:24-37).
#pragma once
#include <stdint.h>

namespace csv {

// majorityVote8 (brick.hpp:24-37) under GNU libstdc++: the unordered_map has
// 13 buckets for <= 8 keys and the identity hash.  Its iteration list holds
// bucket groups newest-group-first and keys newest-first inside a group, and
// max_element keeps the first maximal count.  So among the labels with the
// largest count the winner is the one whose bucket group appeared last and,
// within the group, the label that appeared last.  Positions of first
// appearance stand in for insertion order.
// The common cases come first: one label, or two (on a 4-4 tie the later one: its key
// and, if its bucket is another, its group came last).  Buckets are computed only when
// more labels tie.
__device__ __forceinline__ uint32_t mod13(uint64_t v) {  // 2^32 mod 13 is 9
    return (((uint32_t)(v >> 32) % 13u) * 9u + (uint32_t)v % 13u) % 13u;
}
__device__ __forceinline__ uint64_t majority8(const uint64_t v[8], bool& all) {
    uint32_t ea = 1u;  // which are v[0]
#pragma unroll
    for (int i = 1; i < 8; ++i) ea |= (v[i] == v[0] ? 1u : 0u) << i;
    all = ea == 0xFFu;
    if (all) return v[0];
    uint64_t b = v[7];  // the first that is not v[0]
#pragma unroll
    for (int i = 6; i >= 1; --i)
        if (!((ea >> i) & 1u)) b = v[i];
    uint32_t eb = 0;
#pragma unroll
    for (int i = 1; i < 8; ++i) eb |= (v[i] == b ? 1u : 0u) << i;
    if ((ea | eb) == 0xFFu) return __popc(ea) > 4 ? v[0] : b;
    uint32_t e[8];  // the places of each one's label; 0 but at its first
    uint32_t most = 0, ties = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        uint32_t m = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) m |= (v[j] == v[i] ? 1u : 0u) << j;
        e[i] = (m & ((1u << i) - 1u)) ? 0u : m;
        most = max(most, (uint32_t)__popc(e[i]));
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) ties |= (__popc(e[i]) == (int)most ? 1u : 0u) << i;
    uint32_t best = __ffs(ties) - 1;
    if (ties & (ties - 1)) {
        uint32_t score = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if ((ties >> i) & 1u) {
                const uint32_t bi = mod13(v[i]);
                uint32_t grp = i;
#pragma unroll
                for (int j = 7; j >= 0; --j)
                    if (j < i && e[j] && mod13(v[j]) == bi) grp = j;
                if (8 * grp + i + 1 > score) {
                    score = 8 * grp + i + 1;
                    best = i;
                }
            }
    }
    uint64_t r = v[0];
#pragma unroll
    for (int i = 1; i < 8; ++i)
        if (best == (uint32_t)i) r = v[i];
    return r;
}

}  // namespace csv
