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
// The common cases come first: one label, two (on a 4-4 tie the later one: its key
// and, if its bucket is another, its group came last), three; buckets are computed
// only when labels tie.
__device__ __forceinline__ uint32_t mod13(uint64_t v) {  // 2^32 mod 13 is 9
    return (((uint32_t)(v >> 32) % 13u) * 9u + (uint32_t)v % 13u) % 13u;
}
__device__ __forceinline__ uint32_t places_of(const uint64_t v[8], uint64_t label) {  // bit i: v[i] is it
    uint32_t m = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) m |= (v[i] == label ? 1u : 0u) << i;
    return m;
}
__device__ __forceinline__ uint64_t pick8(const uint64_t v[8], uint32_t at) {
    uint64_t r = v[0];
#pragma unroll
    for (int i = 1; i < 8; ++i)
        if (at == (uint32_t)i) r = v[i];
    return r;
}
__device__ __forceinline__ bool uniform8(const uint64_t v[8]) {
    uint64_t d = 0;
#pragma unroll
    for (int i = 1; i < 8; ++i) d |= v[i] ^ v[0];
    return d == 0;
}
// Any number of labels.
static __device__ __noinline__ uint64_t majority8_any(uint64_t v0, uint64_t v1, uint64_t v2, uint64_t v3, uint64_t v4,
                                                      uint64_t v5, uint64_t v6, uint64_t v7) {
    const uint64_t v[8] = {v0, v1, v2, v3, v4, v5, v6, v7};
    uint32_t e[8];  // the places of each one's label; 0 but at its first
    uint32_t most = 0, best = 0, score = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const uint32_t m = places_of(v, v[i]);
        e[i] = (m & ((1u << i) - 1u)) ? 0u : m;
        most = max(most, (uint32_t)__popc(e[i]));
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
        if (__popc(e[i]) == (int)most) {
            const uint32_t bucket = mod13(v[i]);
            uint32_t grp = i;
#pragma unroll
            for (int j = 7; j >= 0; --j)
                if (j < i && e[j] && mod13(v[j]) == bucket) grp = j;
            if (8 * grp + i + 1 > score) {
                score = 8 * grp + i + 1;
                best = i;
            }
        }
    return pick8(v, best);
}
__device__ __forceinline__ uint64_t majority8_mixed(const uint64_t v[8]) {
    const uint32_t ea = places_of(v, v[0]);
    const uint64_t b = pick8(v, (__ffs(~ea) - 1) & 7u);
    const uint32_t eb = places_of(v, b);
    uint32_t rest = 0xFFu & ~(ea | eb);
    if (!rest) return __popc(ea) > 4 ? v[0] : b;
    const uint64_t c = pick8(v, __ffs(rest) - 1);
    const uint32_t ec = places_of(v, c);
    if (rest & ~ec) return majority8_any(v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7]);
    const int na = __popc(ea), nb = __popc(eb), nc = __popc(ec), most = max(na, max(nb, nc));
    const bool ta = na == most, tb = nb == most, tc = nc == most;
    if (ta + tb + tc == 1) return ta ? v[0] : (tb ? b : c);
    // the keys in order of appearance are 0, 1, 2; a key's group is the first key of its bucket
    const uint32_t ba = mod13(v[0]), bb = mod13(b), bc = mod13(c);
    const int sb = (bb == ba ? 0 : 4) + 1, sc = (bc == ba ? 0 : (bc == bb ? 4 : 8)) + 2;
    if (tc && (!tb || sc > sb)) return c;
    return tb ? b : v[0];
}
__device__ __forceinline__ uint64_t majority8(const uint64_t v[8], bool& all) {
    all = uniform8(v);
    return all ? v[0] : majority8_mixed(v);
}

}  // namespace csv
