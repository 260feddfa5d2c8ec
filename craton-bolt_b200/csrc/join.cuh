// join.cuh — hash join table shared by the probe and the fused join GROUP BY.
#pragma once

#include "ctx.cuh"

// A build-side hash table in the context arena (log2cap >= 6). Slot i holds
// two words:
//   word 0: bitwise NOT of the key (0 = empty; key -1 lives in slot `cap`),
//   word 1: (build row << 32) | u32 payload — or, in a multi-match table
//           (duplicate build keys), (first position in sorted_rows << 32) |
//           number of build rows with the key.
struct bolt_join_table {
    ull* slots = nullptr;
    int32_t log2cap = 0;
    int32_t key_dtype = BOLT_I64;
    int32_t has_payload = 0;
    int32_t multi = 0;                 // 1: duplicate build keys, word 1 as above
    uint32_t* sorted_rows = nullptr;   // multi: the non-NULL build rows, stably sorted by key
    uint64_t n_build = 0;
    uint64_t pinned_mark = 0;  // arena_pinned before this table was placed
    bolt_ctx* owner = nullptr;
};

namespace bolt {

constexpr ull JOIN_HASH = 0x9E3779B97F4A7C15ull;

// A key's home is the first slot of the aligned pair (32 bytes, one sector)
// that its hash picks, and its chain goes on slot by slot from there. A lookup
// step reads a pair at once, so the lanes of a warp, which wait for the
// longest of their chains, go fewer rounds than with single slots (20M probes
// of 1M keys 337 -> 303 us). Blocks of four slots were slower (336 us; 200M
// probes of a 512 MB table 8.0 ms against 4.5: every sector asked for of a
// line costs DRAM as much as the first), and so were tables of 4/3 slots per
// key (0.7M keys 401 -> 627 us).
constexpr int JOIN_BLOCK = 2;
__device__ __forceinline__ ull join_home(ull stored, int log2cap) {
    return ((stored * JOIN_HASH) >> (64 - log2cap)) & ~(ull)(JOIN_BLOCK - 1);
}

struct JoinBlock {
    ull k[JOIN_BLOCK], v[JOIN_BLOCK];
};
// The pair at slot h (even), in one 32-byte load.
__device__ __forceinline__ JoinBlock join_block(const ull* slots, ull h) {
    JoinBlock b;
    asm("ld.global.nc.v4.u64 {%0, %1, %2, %3}, [%4];"
        : "=l"(b.k[0]), "=l"(b.v[0]), "=l"(b.k[1]), "=l"(b.v[1])
        : "l"(slots + 2 * h));
    return b;
}

// One step of a lookup: true when the block settles it, with word 1 of the
// slot, or ~0 when the key is absent, in w.
__device__ __forceinline__ bool join_step(const JoinBlock& b, ull stored, ull& w) {
    bool open = true;  // no empty slot
    w = ~0ull;
#pragma unroll
    for (int i = 0; i < JOIN_BLOCK; ++i) {
        if (b.k[i] == stored) w = b.v[i];
        open = open && b.k[i] != 0;
    }
    return w != ~0ull || !open;
}

// Looks up `key` (already widened to 64 bits); returns word 1 of the slot or
// ~0 when absent (no word 1 is ~0: a build row is below 2^32 - 1). Probes are
// bounded by the table size.
__device__ __forceinline__ ull join_lookup(const ull* slots, int log2cap, ull key) {
    const ull cap = 1ull << log2cap;
    const ull stored = ~key;
    if (stored == 0) {
        const ull* sp = slots + 2 * cap;
        return sp[0] ? sp[1] : ~0ull;
    }
    ull h = join_home(stored, log2cap), w;
    for (ull i = 0; i < cap; i += JOIN_BLOCK) {
        if (join_step(join_block(slots, h), stored, w)) return w;
        h = (h + JOIN_BLOCK) & (cap - 1);
    }
    return ~0ull;
}

}  // namespace bolt
