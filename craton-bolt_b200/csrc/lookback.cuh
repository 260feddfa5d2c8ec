// lookback.cuh — decoupled look-back over 64-bit (status, value) words, one
// word per tile, by a whole warp (Merrill & Garland 2016).
#pragma once

#include "common.cuh"

namespace bolt {

constexpr ull LB_AGG = 1ull << 62;             // the value is the tile's own count
constexpr ull LB_INC = 2ull << 62;             // the value includes every earlier tile
constexpr ull LB_VAL = (1ull << 62) - 1;
constexpr uint32_t LB_SPIN_LIMIT64 = 1u << 22;

// Publishes the tile's count and returns the sum of every earlier tile's, in
// all lanes; then publishes the inclusive sum. Hundreds of tiles are in
// flight at once, so the walk back to the nearest inclusive word is long: the
// warp reads 32 words a round (join probe of 20M rows: one lane reading a
// word at a time 401 us, this 305 us; 128 words a round 377 us, the polls get
// in each other's way). Whole warp. The spin is bounded; on giving up it
// raises ST_FLAG_TIMEOUT and returns what it has.
__device__ __forceinline__ ull warp_look_back(ull* words, uint32_t tile, ull local, uint32_t* status) {
    const int lane = (int)lane_id();
    volatile ull* my = words + tile;
    if (lane == 0) *my = (tile == 0 ? LB_INC : LB_AGG) | local;
    if (tile == 0) return 0;
    ull excl = 0;
    int64_t t = (int64_t)tile - 1;
    uint32_t spins = 0;
    while (t >= 0) {
        const int64_t at = t - lane;
        const ull v = at >= 0 ? ld_volatile(words + at) : LB_INC;
        const uint32_t st = (uint32_t)(v >> 62);
        const uint32_t inc = __ballot_sync(0xffffffffu, st == 2);
        const uint32_t none = __ballot_sync(0xffffffffu, st == 0);
        // Lanes to add: through the nearest inclusive word, or up to the
        // first tile that has published nothing.
        const int f = inc ? __ffs(inc) - 1 : 32, g = none ? __ffs(none) - 1 : 32;
        const int take = f < g ? f + 1 : g;
        ull x = lane < take ? v & LB_VAL : 0ull;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        excl += x;
        if (f < g) break;
        t -= take;
        if (none) {
            if (++spins > LB_SPIN_LIMIT64) {
                if (lane == 0) atomicOr(status, ST_FLAG_TIMEOUT);
                break;
            }
            if (spins > 4) __nanosleep(64);
        }
    }
    if (lane == 0) *my = LB_INC | (excl + local);
    return excl;
}

}  // namespace bolt
