// compact.cu — single-pass filter compaction with decoupled look-back.
//
// Replaces gpu_compact::compact_columns_on_gpu / prefix_scan_mask
// (src/exec/gpu_compact.rs:415,1005) and its kernels (prefix_scan.rs:175,
// 430,834,1227; scan_kernel.rs:265): a predicate kernel writing a u8 mask,
// a per-block scan, block sums scanned on the host (or a look-back with a
// 2-bit status / 30-bit value word) and one gather launch per column.
//
// Here one kernel per call: each CTA takes the next tile in arrival order,
// evaluates the WHERE conjunction (or reads the mask), ranks the kept rows
// with warp ballots in row order, obtains the tile's output offset by
// decoupled look-back over 64-bit (status, value) words, and writes every
// output column. Kept rows of one warp round land on consecutive output
// positions, so the writes are coalesced without staging.
//
// Two kernels share that structure. compact_bulk_kernel (columns that start
// on 16-byte boundaries, the usual case) has one thread stage every column's
// tile into shared memory with bulk copies (cp.async.bulk) completing on an
// mbarrier, and evaluates the WHERE conjuncts on the staged values.
// compact_kernel handles everything else (unaligned columns, wide rows,
// row-id lists) with per-element asynchronous copies or direct loads. The
// NULL split of ORDER BY has kernels of its own (split_count_kernel,
// split_write_kernel).
//
// Large bulk-staged inputs take a two-pass form instead: in one pass a CTA
// waits for its predecessors' counts, and while warp 0 looks back the other
// warps and the tile's memory traffic stand still. compact_count_kernel
// counts each tile's kept rows from the WHERE columns (or the mask) alone,
// compact_scan_kernel turns the counts into tile offsets, and
// compact_bulk_kernel<.., true> stages, ranks and writes every tile with no
// wait on another CTA. The cost is a second read of the WHERE columns
// (4 of the 28 bytes per row of a five-column filter).
#include "compact.cuh"

#include "bulk.cuh"
#include "lookback.cuh"

#include <algorithm>

namespace bolt {
namespace {

constexpr int CP_BLOCK = 256;
constexpr int CP_NW = CP_BLOCK / 32;
// Rows per thread: 8 when columns are read straight from global memory, 4
// when they are staged (smaller tiles keep more CTAs resident per SM).
constexpr int CP_ITEMS_DIRECT = 8;
constexpr int CP_ITEMS_STAGED = 4;
// Largest staged tile (bytes of shared memory per CTA).
constexpr uint32_t CP_STAGE_MAX = 48u << 10;
// Bulk-staged kernels: rows per thread by row width (bytes), and the largest
// stage. Small tiles keep many CTAs (and their copies) in flight per SM.
constexpr int CB_ITEMS_NARROW = 4;  // row_w <= 64: 1,024-row tiles (the vectorised count assumes 4)
constexpr int CB_ITEMS_WIDE = 2;    // row_w <= 128: 512-row tiles
constexpr uint32_t CB_STAGE_MAX = 64u << 10;
// Inputs from this many rows up take the two-pass form.
constexpr uint64_t CB_TWO_PASS_ROWS = 1ull << 22;
// The same for direct loads (a run-start list from a byte mask, say): its
// tiles are short work, so the look-back bounds it (10M rows: one pass 94 us,
// two 76 us).
constexpr uint64_t CP_TWO_PASS_ROWS = 1ull << 20;

struct CpArgs {
    CompactSpec sp;
    ull* lookback;
    uint32_t* tile_ctr;
    uint32_t* status;
    uint32_t soff[CP_MAX_COLS];  // staged kernels: byte offset of each column's tile in shared memory
    uint32_t row_w;              // bytes per row over all columns
    uint32_t* tile_cnt;          // two-pass form: kept rows per tile (pass 1), then before it in its scan group
    ull* group_tot;              // two-pass form: kept rows of each group of SCAN_TILES tiles
};

// Asynchronous global -> shared copy of one element (4, 8 or 16 bytes; both
// addresses aligned to the size), cached in L1 so the predicate's loads of
// the same rows hit.
__device__ __forceinline__ void cp_async_elem(void* dst, const void* src, int width) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    switch (width) {
    case 4: asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory"); break;
    case 8: asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory"); break;
    default: asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory"); break;
    }
}

__device__ __forceinline__ bool cp_cmp_f(double v, int cmp, double lit) {
    switch (cmp) {
    case BOLT_CMP_LT: return v < lit;
    case BOLT_CMP_LE: return v <= lit;
    case BOLT_CMP_GT: return v > lit;
    case BOLT_CMP_GE: return v >= lit;
    case BOLT_CMP_EQ: return v == lit;
    default: return v != lit;
    }
}

__device__ __forceinline__ bool cp_cmp_i(ll v, int cmp, ll lit) {
    switch (cmp) {
    case BOLT_CMP_LT: return v < lit;
    case BOLT_CMP_LE: return v <= lit;
    case BOLT_CMP_GT: return v > lit;
    case BOLT_CMP_GE: return v >= lit;
    case BOLT_CMP_EQ: return v == lit;
    default: return v != lit;
    }
}

__device__ __forceinline__ bool cp_pred(const CompactPred& d, uint64_t r) {
    if (!bit_valid(d.valid, r)) return false;
    if (d.dtype == BOLT_F64 || d.dtype == BOLT_F32) {
        double v = d.dtype == BOLT_F64 ? __ldg((const double*)d.col + r) : (double)__ldg((const float*)d.col + r);
        return cp_cmp_f(v, d.cmp, d.lit_f);
    }
    ll v = d.dtype == BOLT_I32 ? (ll)__ldg((const int32_t*)d.col + r) : __ldg((const ll*)d.col + r);
    return cp_cmp_i(v, d.cmp, d.lit_i);
}

// The same conjunct on a value staged in shared memory (element i of the
// column's tile starting at `st`); the validity bit is read at row r.
__device__ __forceinline__ bool cp_pred_staged(const CompactPred& d, const unsigned char* st, uint32_t i, uint64_t r) {
    if (!bit_valid(d.valid, r)) return false;
    switch (d.dtype) {
    case BOLT_F64: return cp_cmp_f(reinterpret_cast<const double*>(st)[i], d.cmp, d.lit_f);
    case BOLT_F32: return cp_cmp_f((double)reinterpret_cast<const float*>(st)[i], d.cmp, d.lit_f);
    case BOLT_I64: return cp_cmp_i(reinterpret_cast<const ll*>(st)[i], d.cmp, d.lit_i);
    default: return cp_cmp_i((ll)reinterpret_cast<const int32_t*>(st)[i], d.cmp, d.lit_i);
    }
}

// A conjunct split in two so a thread can issue all of its loads before
// the first comparison: the raw 64-bit image of row r's value (integers
// sign-extended, floats as f64 bits), then the comparison on it.
__device__ __forceinline__ ull cp_raw(const CompactPred& d, uint64_t r) {
    switch (d.dtype) {
    case BOLT_F64: return (ull)__ldg((const ll*)d.col + r);
    case BOLT_F32: return (ull)__double_as_longlong((double)__ldg((const float*)d.col + r));
    case BOLT_I64: return (ull)__ldg((const ll*)d.col + r);
    default: return (ull)(ll)__ldg((const int32_t*)d.col + r);
    }
}
__device__ __forceinline__ bool cp_test_raw(const CompactPred& d, ull raw) {
    if (d.dtype == BOLT_F64 || d.dtype == BOLT_F32) return cp_cmp_f(__longlong_as_double((ll)raw), d.cmp, d.lit_f);
    return cp_cmp_i((ll)raw, d.cmp, d.lit_i);
}

// Run by warp 0 once the per-(round, warp) kept counts of the tile are in
// cnt: turns them into row-major exclusive offsets within the tile and
// returns the tile's kept count.
template <int ITEMS>
__device__ __forceinline__ uint32_t cp_tile_scan(uint32_t (*cnt)[CP_NW]) {
    const int lane = threadIdx.x & 31;
    uint32_t local = 0;
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        const uint32_t v = lane < CP_NW ? cnt[j][lane] : 0;
        uint32_t x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        const uint32_t tot = __shfl_sync(0xffffffffu, x, 31);
        if (lane < CP_NW) cnt[j][lane] = local + x - v;
        local += tot;
    }
    return local;
}

// Two-pass form: output offset of `tile` (and, in *total, of everything)
// from the scanned counts: the totals of the earlier groups, added up by the
// warp, and the offset within its group. Run by a whole warp.
constexpr uint32_t SCAN_TILES = 4096;
__device__ __forceinline__ ull cp_two_base(const CpArgs& a, uint32_t tile, uint32_t ntiles, ull* total) {
    const uint32_t lane = lane_id(), g = tile / SCAN_TILES, ng = (ntiles + SCAN_TILES - 1) / SCAN_TILES;
    ull before = 0, all = 0;
    for (uint32_t i = lane; i < (total ? ng : g); i += 32) {
        const ull v = a.group_tot[i];
        all += v;
        if (i < g) before += v;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        before += __shfl_xor_sync(0xffffffffu, before, o);
        if (total) all += __shfl_xor_sync(0xffffffffu, all, o);
    }
    if (total) *total = all;
    return before + a.tile_cnt[tile];
}

// Scans the tile's counts in cnt, leaves its offset `base` (cp_two_base,
// found while the tile's rows were on their way) in *s_base; the last tile
// stores the total.
template <int ITEMS>
__device__ __forceinline__ void cp_two_offsets(const CpArgs& a, uint32_t tile, uint32_t ntiles, uint32_t (*cnt)[CP_NW],
                                               ull base, ull* s_base) {
    const uint32_t local = cp_tile_scan<ITEMS>(cnt);
    if (lane_id() != 0) return;
    *s_base = base;
    if (tile == ntiles - 1) {
        *a.sp.n_out_dev = base + local;
        if (base + local > a.sp.out_cap) atomicOr(a.status, ST_FLAG_CAPACITY);
    }
}

// Run by warp 0 after the tile's counts are in cnt: cp_tile_scan, then the
// look-back over the earlier tiles for the tile's output offset, left in *s_base.
// The last tile stores the total kept count.
template <int ITEMS>
__device__ __forceinline__ void cp_tile_offsets(const CpArgs& a, uint32_t tile, uint32_t ntiles,
                                                uint32_t (*cnt)[CP_NW], ull* s_base) {
    const uint32_t local = cp_tile_scan<ITEMS>(cnt);
    const ull excl = warp_look_back(a.lookback, tile, local, a.status);
    if ((threadIdx.x & 31) != 0) return;
    *s_base = excl;
    if (tile == ntiles - 1) {
        const ull total = excl + local;
        *a.sp.n_out_dev = total;
        if (total > a.sp.out_cap) atomicOr(a.status, ST_FLAG_CAPACITY);
    }
}

// STAGED: every thread first issues asynchronous copies of its rows of every
// output column into shared memory, so the column reads are in flight while
// the predicate is evaluated and the tile's offset is looked back; the
// scatter then reads them back (each thread only its own rows). TWO: the
// two-pass form's second pass, as below.
template <bool STAGED, bool TWO>
__global__ void __launch_bounds__(CP_BLOCK) compact_kernel(const __grid_constant__ CpArgs a) {
    constexpr int CP_ITEMS = STAGED ? CP_ITEMS_STAGED : CP_ITEMS_DIRECT;
    constexpr int CP_TILE = CP_BLOCK * CP_ITEMS;
    extern __shared__ __align__(16) unsigned char cp_stage[];
    __shared__ uint32_t s_tile;
    __shared__ uint32_t cnt[CP_ITEMS][CP_NW];
    __shared__ ull s_base;
    const CompactSpec& sp = a.sp;
    const uint64_t n = sp.n;
    const uint32_t ntiles = (uint32_t)((n + CP_TILE - 1) / CP_TILE);
    if (threadIdx.x == 0) s_tile = TWO ? blockIdx.x : atomicAdd(a.tile_ctr, 1u);
    __syncthreads();
    const uint32_t tile = s_tile;
    if (tile >= ntiles) return;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint64_t base = (uint64_t)tile * CP_TILE;
    if (STAGED) {
#pragma unroll
        for (int j = 0; j < CP_ITEMS; ++j) {
            const uint64_t e = base + (uint64_t)j * CP_BLOCK + threadIdx.x;
            if (e >= n) continue;
            const uint32_t slot = (uint32_t)j * CP_BLOCK + threadIdx.x;
            for (int c = 0; c < sp.n_cols; ++c) {
                const int wd = sp.col[c].width;
                cp_async_elem(cp_stage + a.soff[c] + slot * (uint32_t)wd,
                              static_cast<const unsigned char*>(sp.col[c].in) + e * (uint64_t)wd, wd);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }

    ull tbase0 = 0;
    if (TWO && w == 0) tbase0 = cp_two_base(a, tile, ntiles, nullptr);
    uint32_t keep = 0;  // bit j: element base + j*BLOCK + tid is kept
#pragma unroll
    for (int j = 0; j < CP_ITEMS; ++j) {
        const uint64_t e = base + (uint64_t)j * CP_BLOCK + threadIdx.x;
        bool k = e < n;
        if (k) {
            if (sp.mask) k = sp.mask[e] != 0;
            if (sp.keep_valid_of) k = k && bit_valid(sp.keep_valid_of, e);
            for (int q = 0; q < sp.n_pred; ++q) k = k && cp_pred(sp.pred[q], e);
        }
        const uint32_t b = __ballot_sync(0xffffffffu, k && e < n);
        if (lane == 0) cnt[j][w] = __popc(b);
        if (k && e < n) keep |= 1u << j;
    }
    __syncthreads();
    if (w == 0) {
        if (TWO) {
            cp_two_offsets<CP_ITEMS>(a, tile, ntiles, cnt, tbase0, &s_base);
        } else {
            cp_tile_offsets<CP_ITEMS>(a, tile, ntiles, cnt, &s_base);
        }
    }
    __syncthreads();
    if (STAGED) asm volatile("cp.async.wait_all;" ::: "memory");
    const ull tbase = s_base;
    // Output row of each of this thread's kept rows (~0 when not kept or
    // beyond the output capacity).
    ull pos[CP_ITEMS];
#pragma unroll
    for (int j = 0; j < CP_ITEMS; ++j) {
        const uint32_t b = __ballot_sync(0xffffffffu, (keep >> j) & 1u);
        pos[j] = ~0ull;
        if ((keep >> j) & 1u) {
            const ull at = tbase + cnt[j][w] + __popc(b & lanemask_lt());
            if (at < sp.out_cap) pos[j] = at;
        }
    }
    // Column by column, so the width dispatch runs once per column.
    for (int c = 0; c < sp.n_cols; ++c) {
        const CompactCol& col = sp.col[c];
        const int wd = col.width;
#pragma unroll
        for (int j = 0; j < CP_ITEMS; ++j) {
            if (pos[j] == ~0ull) continue;
            const uint64_t e = base + (uint64_t)j * CP_BLOCK + threadIdx.x;
            const uint32_t slot = (uint32_t)j * CP_BLOCK + threadIdx.x;
            const unsigned char* src = STAGED ? cp_stage + a.soff[c] + slot * (uint32_t)wd
                                              : static_cast<const unsigned char*>(col.in) + e * (uint64_t)wd;
            if (wd == 4) {
                ((uint32_t*)col.out)[pos[j]] = STAGED ? *reinterpret_cast<const uint32_t*>(src)
                                                      : __ldg(reinterpret_cast<const uint32_t*>(src));
            } else if (wd == 8) {
                ((ull*)col.out)[pos[j]] = STAGED ? *reinterpret_cast<const ull*>(src)
                                                 : __ldg(reinterpret_cast<const ull*>(src));
            } else {
                ((ulonglong2*)col.out)[pos[j]] = STAGED ? *reinterpret_cast<const ulonglong2*>(src)
                                                        : __ldg(reinterpret_cast<const ulonglong2*>(src));
            }
            if (col.out_valid && bit_valid(col.in_valid, e)) set_bit_atomic(col.out_valid, pos[j], true);
        }
    }
    if (sp.row_ids) {
#pragma unroll
        for (int j = 0; j < CP_ITEMS; ++j) {
            if (pos[j] == ~0ull) continue;
            const uint64_t e = base + (uint64_t)j * CP_BLOCK + threadIdx.x;
            sp.row_ids[pos[j]] = (uint32_t)e + sp.row_id_base;
        }
    }
}

// Bulk-staged compaction (every column starts on a 16-byte boundary; no
// keep_valid_of selection). Thread 0 issues one bulk copy per
// column of the tile's TILE rows (TILE * width bytes, a multiple of 16) into
// shared memory, completing on one mbarrier; the last, partial tile is
// copied element by element instead. Ranking, look-back and scatter follow
// compact_kernel, reading the staged values. TWO: the two-pass form's second
// pass (CTA i takes tile i; its offset comes from compact_scan_kernel).
template <int ITEMS, bool TWO>
__global__ void __launch_bounds__(CP_BLOCK) compact_bulk_kernel(const __grid_constant__ CpArgs a) {
    constexpr int TILE = CP_BLOCK * ITEMS;
    extern __shared__ __align__(128) unsigned char stg[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t s_tile;
    __shared__ uint32_t cnt[ITEMS][CP_NW];
    __shared__ ull s_base;
    const CompactSpec& sp = a.sp;
    const uint64_t n = sp.n;
    const uint32_t ntiles = (uint32_t)((n + TILE - 1) / TILE);
    if (threadIdx.x == 0) {
        s_tile = TWO ? blockIdx.x : atomicAdd(a.tile_ctr, 1u);
        mbar_init(&bar, 1);
        mbar_init_fence();
    }
    __syncthreads();
    const uint32_t tile = s_tile;
    if (tile >= ntiles) return;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint64_t base = (uint64_t)tile * TILE;
    const uint32_t rows = (n - base) < (uint64_t)TILE ? (uint32_t)(n - base) : (uint32_t)TILE;
    const bool whole = rows == (uint32_t)TILE;
    bool ok = true;
    ull tbase0 = 0;
    if (whole) {
        if (threadIdx.x == 0) {
            mbar_arrive_expect_tx(&bar, (uint32_t)TILE * a.row_w);
            const uint64_t pol = l2_evict_first_policy();
            for (int c = 0; c < sp.n_cols; ++c) {
                const uint32_t wd = (uint32_t)sp.col[c].width;
                bulk_load(stg + a.soff[c], static_cast<const unsigned char*>(sp.col[c].in) + base * wd,
                          (uint32_t)TILE * wd, &bar, pol);
            }
        }
        if (TWO && w == 0) {
            __syncwarp();
            tbase0 = cp_two_base(a, tile, ntiles, nullptr);
        }
        ok = mbar_wait(&bar, 0);
    } else {
        for (int c = 0; c < sp.n_cols; ++c) {
            const int wd = sp.col[c].width;
            const unsigned char* src = static_cast<const unsigned char*>(sp.col[c].in) + base * (uint64_t)wd;
            unsigned char* dst = stg + a.soff[c];
            for (uint32_t i = threadIdx.x; i < rows; i += CP_BLOCK) {
                if (wd == 4) reinterpret_cast<uint32_t*>(dst)[i] = __ldg(reinterpret_cast<const uint32_t*>(src) + i);
                else if (wd == 8) reinterpret_cast<ull*>(dst)[i] = __ldg(reinterpret_cast<const ull*>(src) + i);
                else reinterpret_cast<ulonglong2*>(dst)[i] = __ldg(reinterpret_cast<const ulonglong2*>(src) + i);
            }
        }
        if (TWO && w == 0) tbase0 = cp_two_base(a, tile, ntiles, nullptr);
        __syncthreads();
    }
    if (!ok && threadIdx.x == 0) atomicOr(a.status, ST_FLAG_TIMEOUT);

    // A tile whose copy did not complete keeps no rows (the call reports
    // TIMEOUT) but still publishes its count, so later tiles finish.
    uint32_t keep = 0;
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        const uint32_t i = (uint32_t)j * CP_BLOCK + threadIdx.x;
        const uint64_t e = base + i;
        bool k = ok && i < rows;
        if (k) {
            if (sp.mask) k = sp.mask[e] != 0;
            for (int q = 0; q < sp.n_pred; ++q) k = k && cp_pred_staged(sp.pred[q], stg + a.soff[sp.pred[q].col_idx], i, e);
        }
        k = k && ok && i < rows;
        const uint32_t b = __ballot_sync(0xffffffffu, k);
        if (lane == 0) cnt[j][w] = __popc(b);
        if (k) keep |= 1u << j;
    }
    __syncthreads();
    if (w == 0) {
        if (TWO) {
            cp_two_offsets<ITEMS>(a, tile, ntiles, cnt, tbase0, &s_base);
        } else {
            cp_tile_offsets<ITEMS>(a, tile, ntiles, cnt, &s_base);
        }
    }
    __syncthreads();
    const ull tbase = s_base;
    ull pos[ITEMS];
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        const uint32_t b = __ballot_sync(0xffffffffu, (keep >> j) & 1u);
        pos[j] = ~0ull;
        if ((keep >> j) & 1u) {
            const ull at = tbase + cnt[j][w] + __popc(b & lanemask_lt());
            if (at < sp.out_cap) pos[j] = at;
        }
    }
    for (int c = 0; c < sp.n_cols; ++c) {
        const CompactCol& col = sp.col[c];
        const int wd = col.width;
        const unsigned char* st = stg + a.soff[c];
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
            if (pos[j] == ~0ull) continue;
            const uint32_t i = (uint32_t)j * CP_BLOCK + threadIdx.x;
            if (wd == 4) ((uint32_t*)col.out)[pos[j]] = reinterpret_cast<const uint32_t*>(st)[i];
            else if (wd == 8) ((ull*)col.out)[pos[j]] = reinterpret_cast<const ull*>(st)[i];
            else ((ulonglong2*)col.out)[pos[j]] = reinterpret_cast<const ulonglong2*>(st)[i];
            if (col.out_valid && bit_valid(col.in_valid, base + i)) set_bit_atomic(col.out_valid, pos[j], true);
        }
    }
    if (sp.row_ids) {
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
            if (pos[j] == ~0ull) continue;
            sp.row_ids[pos[j]] = (uint32_t)(base + (uint32_t)j * CP_BLOCK + threadIdx.x) + sp.row_id_base;
        }
    }
    // A copy that missed its wait may still be landing: wait for it (again
    // bounded) before the CTA's shared memory can be handed to another CTA.
    if (!ok && threadIdx.x == 0) mbar_wait(&bar, 0);
}

// Two-pass form, pass 1: kept rows of each tile of CP_BLOCK * ITEMS rows,
// from the mask or the WHERE columns alone. A CTA takes CC_GROUP tiles at a
// time (grid-stride) and issues every load of a conjunct before comparing.
// VEC: the selection is a byte mask or one Int32 conjunct without a
// validity bitmap, on a 16-byte aligned column: each thread then reads 16
// consecutive rows with 16-byte loads (counts need no row order).
constexpr int CC_GROUP = 4;
template <int ITEMS, bool VEC>
__global__ void __launch_bounds__(CP_BLOCK) compact_count_kernel(const __grid_constant__ CpArgs a) {
    constexpr int TILE = CP_BLOCK * ITEMS;
    constexpr int R = ITEMS * CC_GROUP;  // rows per thread per step
    static_assert(!VEC || CP_BLOCK * 16 == CC_GROUP * TILE, "vectorised count: 16 rows per thread cover the group");
    __shared__ uint32_t wcnt[CC_GROUP][CP_NW];
    const CompactSpec& sp = a.sp;
    const uint64_t n = sp.n;
    const uint32_t ntiles = (uint32_t)((n + TILE - 1) / TILE);
    const uint32_t ngroups = (ntiles + CC_GROUP - 1) / CC_GROUP;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (uint32_t grp = blockIdx.x; grp < ngroups; grp += gridDim.x) {
        const uint64_t base = (uint64_t)grp * CC_GROUP * TILE;
        uint32_t c[CC_GROUP];
#pragma unroll
        for (int g = 0; g < CC_GROUP; ++g) c[g] = 0;
        if (VEC) {
            // Thread t: rows base + 16t .. base + 16t + 15, all inside tile
            // (16t) / TILE of the group.
            const uint64_t r0 = base + (uint64_t)threadIdx.x * 16;
            uint32_t k = 0;
            if (r0 + 16 <= n) {
                if (sp.mask) {
                    const uint4 m = __ldg(reinterpret_cast<const uint4*>(sp.mask + r0));
                    const uint32_t wv[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
                    for (int q = 0; q < 4; ++q)
#pragma unroll
                        for (int b = 0; b < 4; ++b) k += ((wv[q] >> (8 * b)) & 0xFFu) != 0;
                } else {
                    const CompactPred& d = sp.pred[0];
                    const int4* src = reinterpret_cast<const int4*>((const int32_t*)d.col + r0);
                    int4 v[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) v[q] = __ldg(src + q);
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        k += cp_cmp_i(v[q].x, d.cmp, d.lit_i);
                        k += cp_cmp_i(v[q].y, d.cmp, d.lit_i);
                        k += cp_cmp_i(v[q].z, d.cmp, d.lit_i);
                        k += cp_cmp_i(v[q].w, d.cmp, d.lit_i);
                    }
                }
            } else {
                for (uint64_t r = r0; r < n && r < r0 + 16; ++r)
                    k += sp.mask ? (sp.mask[r] != 0) : cp_cmp_i(((const int32_t*)sp.pred[0].col)[r], sp.pred[0].cmp,
                                                              sp.pred[0].lit_i);
            }
            // Warps w = 2g, 2g + 1 cover tile g of the group (TILE = 1024
            // rows = 64 threads x 16) when ITEMS == 4.
            k = __reduce_add_sync(0xffffffffu, k);
            if (lane == 0) wcnt[0][w] = k;
            __syncthreads();
            if (threadIdx.x < CC_GROUP) {
                const uint32_t tile = grp * CC_GROUP + threadIdx.x;
                constexpr int WPT = CP_NW / CC_GROUP;  // warps per tile
                uint32_t t = 0;
#pragma unroll
                for (int i = 0; i < WPT; ++i) t += wcnt[0][threadIdx.x * WPT + i];
                if (tile < ntiles) a.tile_cnt[tile] = t;
            }
            __syncthreads();
            continue;
        }
        uint32_t keep = 0;  // bit j: row base + j*BLOCK + tid
#pragma unroll
        for (int j = 0; j < R; ++j)
            if (base + (uint64_t)j * CP_BLOCK + threadIdx.x < n) keep |= 1u << j;
        if (sp.mask) {
            uint8_t m[R];
#pragma unroll
            for (int j = 0; j < R; ++j) {
                const uint64_t e = base + (uint64_t)j * CP_BLOCK + threadIdx.x;
                m[j] = ((keep >> j) & 1u) ? __ldg(sp.mask + e) : (uint8_t)0;
            }
#pragma unroll
            for (int j = 0; j < R; ++j)
                if (!m[j]) keep &= ~(1u << j);
        }
        for (int q = 0; q < sp.n_pred; ++q) {
            const CompactPred& d = sp.pred[q];
            ull raw[R];
#pragma unroll
            for (int j = 0; j < R; ++j) {
                const uint64_t e = base + (uint64_t)j * CP_BLOCK + threadIdx.x;
                raw[j] = ((keep >> j) & 1u) ? cp_raw(d, e) : 0ull;
            }
#pragma unroll
            for (int j = 0; j < R; ++j) {
                const uint64_t e = base + (uint64_t)j * CP_BLOCK + threadIdx.x;
                if (((keep >> j) & 1u) && !(bit_valid(d.valid, e) && cp_test_raw(d, raw[j]))) keep &= ~(1u << j);
            }
        }
#pragma unroll
        for (int j = 0; j < R; ++j) {
            c[j / ITEMS] += __popc(__ballot_sync(0xffffffffu, (keep >> j) & 1u));
        }
        if (lane == 0) {
#pragma unroll
            for (int g = 0; g < CC_GROUP; ++g) wcnt[g][w] = c[g];
        }
        __syncthreads();
        if (threadIdx.x < CC_GROUP) {
            const uint32_t tile = grp * CC_GROUP + threadIdx.x;
            uint32_t t = 0;
#pragma unroll
            for (int i = 0; i < CP_NW; ++i) t += wcnt[threadIdx.x][i];
            if (tile < ntiles) a.tile_cnt[tile] = t;
        }
        __syncthreads();
    }
}

// Two-pass form: CTA g turns the counts of tiles [g * SCAN_TILES, ...) into
// exclusive offsets within the group, in place, and stores the group's total;
// the scatter pass adds up the earlier groups' totals itself (24 of them for
// 100M rows). One CTA over all 98K counts took 84 us.
__global__ void __launch_bounds__(1024) compact_scan_kernel(const __grid_constant__ CpArgs a, uint32_t ntiles) {
    __shared__ uint32_t wsum[32];
    const int t = threadIdx.x, w = t >> 5, lane = t & 31;
    const uint64_t i = (uint64_t)blockIdx.x * SCAN_TILES + 4 * (uint64_t)t;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (i + 4 <= ntiles) {
        v = *reinterpret_cast<const uint4*>(a.tile_cnt + i);
    } else {
        if (i < ntiles) v.x = a.tile_cnt[i];
        if (i + 1 < ntiles) v.y = a.tile_cnt[i + 1];
        if (i + 2 < ntiles) v.z = a.tile_cnt[i + 2];
    }
    const uint32_t mine = v.x + v.y + v.z + v.w;
    uint32_t x = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) wsum[w] = x;
    __syncthreads();
    const uint32_t ws = wsum[lane];
    const uint32_t before = __reduce_add_sync(0xffffffffu, lane < w ? ws : 0u);
    const uint32_t o0 = before + x - mine, o1 = o0 + v.x, o2 = o1 + v.y, o3 = o2 + v.z;
    if (i + 4 <= ntiles) {
        *reinterpret_cast<uint4*>(a.tile_cnt + i) = make_uint4(o0, o1, o2, o3);
    } else {
        if (i < ntiles) a.tile_cnt[i] = o0;
        if (i + 1 < ntiles) a.tile_cnt[i + 1] = o1;
        if (i + 2 < ntiles) a.tile_cnt[i + 2] = o2;
    }
    if (t == 1023) a.group_tot[blockIdx.x] = o3 + v.w;
}

// NULL split: the rows' ids (ids_in[e], or e) parted into the valid ones and
// the NULL ones, each in input order. The validity bits of permuted rows are
// random bytes of the bitmap, which is what a split waits for, so they are
// gathered once: this pass packs them in element order and counts each
// 2,048-row tile's, and split_write_kernel places both parts from the packed
// bits. (Two compactions, each gathering in both of its passes: 257 us for
// for 10M rows.) Without room for the packed bits (PACKED false) the second
// pass gathers them again.
template <bool PACKED>
__global__ void __launch_bounds__(CP_BLOCK) split_count_kernel(const __grid_constant__ CpArgs a, const uint32_t* ids_in,
                                                               uint32_t* bits) {
    constexpr int TILE = CP_BLOCK * CP_ITEMS_DIRECT;
    __shared__ uint32_t wcnt[CP_NW];
    const CompactSpec& sp = a.sp;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint64_t base = (uint64_t)blockIdx.x * TILE;
    uint32_t id[CP_ITEMS_DIRECT];
#pragma unroll
    for (int j = 0; j < CP_ITEMS_DIRECT; ++j) {
        const uint64_t e = base + (uint64_t)j * CP_BLOCK + threadIdx.x;
        id[j] = e < sp.n ? (ids_in ? __ldg(ids_in + e) : (uint32_t)e) : 0u;
    }
    uint32_t c = 0;
#pragma unroll
    for (int j = 0; j < CP_ITEMS_DIRECT; ++j) {
        const uint64_t e = base + (uint64_t)j * CP_BLOCK + threadIdx.x;
        const uint32_t m = __ballot_sync(0xffffffffu, e < sp.n && bit_valid(sp.keep_valid_of, id[j]));
        if (PACKED && lane == 0) bits[e >> 5] = m;  // (whole tiles of words are allocated)
        c += __popc(m);
    }
    if (lane == 0) wcnt[w] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0;
#pragma unroll
        for (int i = 0; i < CP_NW; ++i) t += wcnt[i];
        a.tile_cnt[blockIdx.x] = t;
    }
}

// sp.row_ids receives the valid ids; `nulls` the others, from row 0
// (nulls_first) or from the number of valid rows.
template <bool PACKED>
__global__ void __launch_bounds__(CP_BLOCK) split_write_kernel(const __grid_constant__ CpArgs a, const uint32_t* ids_in,
                                                               const uint32_t* bits, uint32_t* nulls, int nulls_first, uint32_t ntiles) {
    constexpr int TILE = CP_BLOCK * CP_ITEMS_DIRECT, WORDS = TILE / 32;
    __shared__ uint32_t word[WORDS], pre[WORDS];
    __shared__ ull s_base, s_total;
    const CompactSpec& sp = a.sp;
    const int lane = threadIdx.x & 31;
    const uint32_t tile = blockIdx.x;
    const uint64_t base = (uint64_t)tile * TILE;
    if (!PACKED) {
#pragma unroll
        for (int j = 0; j < CP_ITEMS_DIRECT; ++j) {
            const uint32_t i = (uint32_t)j * CP_BLOCK + threadIdx.x;
            const uint64_t e = base + i;
            const uint32_t m = __ballot_sync(0xffffffffu, e < sp.n && bit_valid(sp.keep_valid_of, ids_in ? __ldg(ids_in + e) : e));
            if (lane == 0) word[i >> 5] = m;
        }
        __syncthreads();
    }
    if (threadIdx.x < 32) {
        ull total;
        const ull b = cp_two_base(a, tile, ntiles, &total);
        uint32_t run = 0;
#pragma unroll
        for (int h = 0; h < WORDS; h += 32) {
            const uint32_t m = PACKED ? bits[base / 32 + h + lane] : word[h + lane], c = __popc(m);
            uint32_t x = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            word[h + lane] = m;
            pre[h + lane] = run + x - c;
            run += __shfl_sync(0xffffffffu, x, 31);
        }
        if (lane == 0) {
            s_base = b;
            s_total = total;
            if (tile == 0) *sp.n_out_dev = total;
        }
    }
    uint32_t id[CP_ITEMS_DIRECT];
#pragma unroll
    for (int j = 0; j < CP_ITEMS_DIRECT; ++j) {
        const uint64_t e = base + (uint64_t)j * CP_BLOCK + threadIdx.x;
        id[j] = e < sp.n ? (ids_in ? __ldg(ids_in + e) : (uint32_t)e) : 0u;
    }
    __syncthreads();
    const ull nb = nulls_first ? 0ull : s_total;
#pragma unroll
    for (int j = 0; j < CP_ITEMS_DIRECT; ++j) {
        const uint32_t i = (uint32_t)j * CP_BLOCK + threadIdx.x;
        const uint64_t e = base + i;
        if (e >= sp.n) continue;
        const uint32_t m = word[i >> 5];
        const ull rank = s_base + pre[i >> 5] + __popc(m & lanemask_lt());
        if ((m >> lane) & 1u) sp.row_ids[rank] = id[j];
        else nulls[nb + (e - rank)] = id[j];
    }
}

}  // namespace

bolt_status compact_enqueue(bolt_ctx* ctx, cudaStream_t s, const CompactSpec& spec, uint32_t flags) {
    CpArgs a{};
    a.sp = spec;
    uint32_t row_w = 0;
    bool aligned = spec.n_cols > 0, al16 = spec.n_cols > 0;
    for (int c = 0; c < spec.n_cols; ++c) {
        const int wd = spec.col[c].width;
        const uintptr_t addr = reinterpret_cast<uintptr_t>(spec.col[c].in);
        aligned = aligned && (wd == 4 || wd == 8 || wd == 16) && addr % (uintptr_t)wd == 0;
        al16 = al16 && addr % 16 == 0;
        row_w += (uint32_t)wd;
    }
    a.row_w = row_w;
    // Bulk-staged tiles: columns on 16-byte boundaries, a tile of them within
    // the stage budget, and a plain selection (no keep_valid_of).
    int bulk_items = 0;
    if (aligned && al16 && !spec.keep_valid_of && !(flags & BOLT_FLAG_KERNEL_REGS)) {
        if (row_w * (uint32_t)(CP_BLOCK * CB_ITEMS_NARROW) <= CB_STAGE_MAX) bulk_items = CB_ITEMS_NARROW;
        else if (row_w * (uint32_t)(CP_BLOCK * CB_ITEMS_WIDE) <= CB_STAGE_MAX) bulk_items = CB_ITEMS_WIDE;
    }
    // Otherwise per-element asynchronous copies when a tile fits the budget
    // and every input is aligned to its width, else direct loads.
    const bool staged = !bulk_items && aligned && row_w * (uint32_t)(CP_BLOCK * CP_ITEMS_STAGED) <= CP_STAGE_MAX;
    const uint32_t items = bulk_items ? (uint32_t)bulk_items : staged ? (uint32_t)CP_ITEMS_STAGED : (uint32_t)CP_ITEMS_DIRECT;
    uint32_t off = 0;
    for (int c = 0; c < spec.n_cols; ++c) {
        a.soff[c] = off;
        off += (uint32_t)spec.col[c].width * (uint32_t)CP_BLOCK * items;
    }
    const uint32_t stage_bytes = row_w * (uint32_t)CP_BLOCK * items;
    const uint64_t tile_rows = (uint64_t)CP_BLOCK * items;
    const uint64_t ntiles = (spec.n + tile_rows - 1) / tile_rows;
    // Large bulk-staged inputs run the two-pass form (no CTA waits on
    // another); the rest run one pass with decoupled look-back.
    const bool two = spec.n >= (bulk_items ? CB_TWO_PASS_ROWS : CP_TWO_PASS_ROWS) && !staged && !spec.keep_valid_of;
    a.tile_ctr = (uint32_t*)arena_alloc(ctx, 64);
    if (two) {
        const uint64_t groups = (ntiles + SCAN_TILES - 1) / SCAN_TILES;
        a.group_tot = (ull*)arena_alloc(ctx, (groups + 1) * 8 + ntiles * 4);
        a.tile_cnt = reinterpret_cast<uint32_t*>(a.group_tot + ((groups + 1) & ~1ull));
        if (!a.group_tot || !a.tile_ctr) return fail(ctx, BOLT_ERR_CAPACITY, "compaction: scratch arena too small");
    } else {
        a.lookback = (ull*)arena_alloc(ctx, (ntiles + 1) * 8);
        if (!a.lookback || !a.tile_ctr) return fail(ctx, BOLT_ERR_CAPACITY, "compaction: scratch arena too small");
        BOLT_CUDA(ctx, cudaMemsetAsync(a.lookback, 0, (ntiles + 1) * 8, s));
    }
    a.status = ctx->d_status;
    BOLT_CUDA(ctx, cudaMemsetAsync(a.tile_ctr, 0, 64, s));
    if (spec.n == 0) {
        BOLT_CUDA(ctx, cudaMemsetAsync(spec.n_out_dev, 0, 8, s));
        return BOLT_OK;
    }
    for (int c = 0; c < spec.n_cols; ++c) {
        const uint64_t rows = spec.out_cap < spec.n ? spec.out_cap : spec.n;
        if (spec.col[c].out_valid) BOLT_CUDA(ctx, cudaMemsetAsync(spec.col[c].out_valid, 0, (rows + 7) / 8, s));
    }
    kernel_mark_begin(ctx, flags, s);
    if (two) {
        const uint64_t ngroups = (ntiles + CC_GROUP - 1) / CC_GROUP;
        const unsigned cg = (unsigned)std::min<uint64_t>(ngroups, (uint64_t)ctx->num_sms * 8);
        const unsigned sgrid = (unsigned)((ntiles + SCAN_TILES - 1) / SCAN_TILES);
        // Vectorised count: a byte mask or one Int32 conjunct without a
        // validity bitmap, on 16-byte boundaries (1,024-row tiles only).
        const bool vec = bulk_items == 4 &&
                         ((spec.mask && spec.n_pred == 0 && reinterpret_cast<uintptr_t>(spec.mask) % 16 == 0) ||
                          (!spec.mask && spec.n_pred == 1 && spec.pred[0].dtype == BOLT_I32 && !spec.pred[0].valid &&
                           reinterpret_cast<uintptr_t>(spec.pred[0].col) % 16 == 0));
        if (!bulk_items) {
            compact_count_kernel<CP_ITEMS_DIRECT, false><<<cg, CP_BLOCK, 0, s>>>(a);
            compact_scan_kernel<<<sgrid, 1024, 0, s>>>(a, (uint32_t)ntiles);
            compact_kernel<false, true><<<(unsigned)ntiles, CP_BLOCK, 0, s>>>(a);
        } else if (bulk_items == CB_ITEMS_NARROW) {
            if (vec) compact_count_kernel<CB_ITEMS_NARROW, true><<<cg, CP_BLOCK, 0, s>>>(a);
            else compact_count_kernel<CB_ITEMS_NARROW, false><<<cg, CP_BLOCK, 0, s>>>(a);
            compact_scan_kernel<<<sgrid, 1024, 0, s>>>(a, (uint32_t)ntiles);
            BOLT_CUDA(ctx, smem_optin(compact_bulk_kernel<CB_ITEMS_NARROW, true>, ctx));
            compact_bulk_kernel<CB_ITEMS_NARROW, true><<<(unsigned)ntiles, CP_BLOCK, stage_bytes, s>>>(a);
        } else {
            compact_count_kernel<CB_ITEMS_WIDE, false><<<cg, CP_BLOCK, 0, s>>>(a);
            compact_scan_kernel<<<sgrid, 1024, 0, s>>>(a, (uint32_t)ntiles);
            BOLT_CUDA(ctx, smem_optin(compact_bulk_kernel<CB_ITEMS_WIDE, true>, ctx));
            compact_bulk_kernel<CB_ITEMS_WIDE, true><<<(unsigned)ntiles, CP_BLOCK, stage_bytes, s>>>(a);
        }
        ctx->last_launches += 2;
    } else if (bulk_items == CB_ITEMS_NARROW) {
        BOLT_CUDA(ctx, smem_optin(compact_bulk_kernel<CB_ITEMS_NARROW, false>, ctx));
        compact_bulk_kernel<CB_ITEMS_NARROW, false><<<(unsigned)ntiles, CP_BLOCK, stage_bytes, s>>>(a);
    } else if (bulk_items == CB_ITEMS_WIDE) {
        BOLT_CUDA(ctx, smem_optin(compact_bulk_kernel<CB_ITEMS_WIDE, false>, ctx));
        compact_bulk_kernel<CB_ITEMS_WIDE, false><<<(unsigned)ntiles, CP_BLOCK, stage_bytes, s>>>(a);
    } else if (staged) {
        BOLT_CUDA(ctx, smem_optin(compact_kernel<true, false>, ctx));
        compact_kernel<true, false><<<(unsigned)ntiles, CP_BLOCK, stage_bytes, s>>>(a);
    } else {
        compact_kernel<false, false><<<(unsigned)ntiles, CP_BLOCK, 0, s>>>(a);
    }
    kernel_mark_end(ctx, flags, s);
    ctx->last_launches++;
    BOLT_CUDA(ctx, cudaGetLastError());
    return BOLT_OK;
}

bolt_status null_split_enqueue(bolt_ctx* ctx, cudaStream_t s, uint64_t n, const uint8_t* valid, const uint32_t* ids_in,
                               uint32_t* valid_ids, uint32_t* nulls, bool nulls_first, ull* n_valid_dev) {
    CpArgs a{};
    a.sp.n = n;
    a.sp.keep_valid_of = valid;
    a.sp.row_ids = valid_ids;
    a.sp.n_out_dev = n_valid_dev;
    a.status = ctx->d_status;
    if (n == 0) {
        BOLT_CUDA(ctx, cudaMemsetAsync(n_valid_dev, 0, 8, s));
        return BOLT_OK;
    }
    constexpr uint64_t TILE = (uint64_t)CP_BLOCK * CP_ITEMS_DIRECT;
    const uint64_t ntiles = (n + TILE - 1) / TILE, groups = (ntiles + SCAN_TILES - 1) / SCAN_TILES;
    const uint64_t mark = ctx->arena_used;  // (scratch of these launches only: later work on the stream may reuse it)
    a.group_tot = (ull*)arena_alloc(ctx, (groups + 1) * 8 + ntiles * 4);
    a.tile_cnt = reinterpret_cast<uint32_t*>(a.group_tot + ((groups + 1) & ~1ull));
    if (!a.group_tot) return fail(ctx, BOLT_ERR_CAPACITY, "NULL split: scratch arena too small");
    // (A column of hardly more than NULLs sorts in little more than its valid
    // ids: the bits may be what does not fit.)
    uint32_t* bits = (uint32_t*)arena_alloc(ctx, ntiles * TILE / 8);
    if (bits) split_count_kernel<true><<<(unsigned)ntiles, CP_BLOCK, 0, s>>>(a, ids_in, bits);
    else split_count_kernel<false><<<(unsigned)ntiles, CP_BLOCK, 0, s>>>(a, ids_in, bits);
    compact_scan_kernel<<<(unsigned)groups, 1024, 0, s>>>(a, (uint32_t)ntiles);
    auto write = bits ? split_write_kernel<true> : split_write_kernel<false>;
    write<<<(unsigned)ntiles, CP_BLOCK, 0, s>>>(a, ids_in, bits, nulls, nulls_first ? 1 : 0, (uint32_t)ntiles);
    ctx->arena_used = mark;
    ctx->last_launches += 3;
    BOLT_CUDA(ctx, cudaGetLastError());
    return BOLT_OK;
}

}  // namespace bolt

using namespace bolt;

namespace {

int width_of(int dt) {
    switch (dt) {
    case BOLT_I32: case BOLT_F32: case BOLT_U32: return 4;
    case BOLT_I64: case BOLT_F64: return 8;
    case BOLT_DEC128: return 16;
    }
    return 0;
}

bolt_status compact_common(bolt_ctx* ctx, const bolt_col_view* cols, int32_t n_cols, const bolt_pred* preds,
                           int32_t n_preds, const uint8_t* mask, bolt_col_mut* out, bolt_col_mut* row_ids,
                           uint64_t* n_out, uint32_t flags, bolt_stream stream) {
    if (!ctx || !n_out || n_cols < 0 || n_cols > CP_MAX_COLS || n_preds < 0 || n_preds > CP_MAX_PREDS)
        return ctx ? fail(ctx, BOLT_ERR_INVALID, "compaction: bad arguments") : BOLT_ERR_INVALID;
    if (n_cols == 0 && !row_ids) return fail(ctx, BOLT_ERR_INVALID, "compaction: nothing to output");
    cudaStream_t s = (cudaStream_t)stream;
    bolt_status st = call_begin(ctx, flags, s);
    if (st != BOLT_OK) return st;
    CompactSpec sp;
    uint64_t n = n_cols > 0 ? cols[0].len : 0;
    if (n_cols == 0 && n_preds > 0) return fail(ctx, BOLT_ERR_INVALID, "compaction: predicates need columns");
    for (int c = 0; c < n_cols; ++c) {
        if (cols[c].len != n) return fail(ctx, BOLT_ERR_INVALID, "compaction: column lengths differ");
        const int wd = width_of(cols[c].dtype);
        if (!wd || !out || out[c].dtype != cols[c].dtype)
            return fail(ctx, BOLT_ERR_INVALID, "compaction: column %d dtype mismatch", c);
        if (!col_aligned(cols[c].data, cols[c].dtype) || !col_aligned(out[c].data, cols[c].dtype))
            return fail(ctx, BOLT_ERR_INVALID, "compaction: column %d is not aligned to its element width", c);
        sp.col[c] = CompactCol{cols[c].data, cols[c].validity, out[c].data, cols[c].validity ? out[c].validity : nullptr, wd};
        sp.out_cap = sp.out_cap < out[c].cap ? sp.out_cap : out[c].cap;
    }
    if (row_ids) {
        if (row_ids->dtype != BOLT_U32) return fail(ctx, BOLT_ERR_INVALID, "compaction: row ids must be U32");
        sp.row_ids = (uint32_t*)row_ids->data;
        sp.out_cap = sp.out_cap < row_ids->cap ? sp.out_cap : row_ids->cap;
    }
    if (n >= (1ull << 32) && row_ids) return fail(ctx, BOLT_DECLINE, "compaction: row ids need n < 2^32");
    sp.n_cols = n_cols;
    sp.n = n;
    sp.mask = mask;
    for (int q = 0; q < n_preds; ++q) {
        if (preds[q].col < 0 || preds[q].col >= n_cols) return fail(ctx, BOLT_ERR_INVALID, "compaction: WHERE column out of range");
        const bolt_col_view& c = cols[preds[q].col];
        if (c.dtype == BOLT_DEC128 || c.dtype == BOLT_U32) return fail(ctx, BOLT_DECLINE, "compaction: WHERE on dtype %d", c.dtype);
        sp.pred[q] = CompactPred{c.data, c.validity, c.dtype, preds[q].cmp, preds[q].lit_i, preds[q].lit_f, preds[q].col};
    }
    sp.n_pred = n_preds;
    ull* cnt = (ull*)arena_alloc(ctx, 256);
    if (!cnt) return fail(ctx, BOLT_ERR_CAPACITY, "compaction: scratch arena too small");
    sp.n_out_dev = cnt;
    st = compact_enqueue(ctx, s, sp, flags);
    if (st != BOLT_OK) return st;
    if (flags & BOLT_FLAG_ASYNC) return call_end(ctx, flags, s);
    uint32_t f = 0;
    st = call_finish(ctx, flags, s, cnt, 1, &f);
    if (st != BOLT_OK) return st;
    *n_out = ctx->h_words[2];
    return flags_to_status(ctx, f, "compaction");
}

}  // namespace

extern "C" bolt_status bolt_compact(bolt_ctx* ctx, const bolt_col_view* cols, int32_t n_cols, const bolt_pred* preds,
                                    int32_t n_preds, bolt_col_mut* out, bolt_col_mut* row_ids, uint64_t* n_out,
                                    uint32_t flags, bolt_stream stream) {
    return compact_common(ctx, cols, n_cols, preds, n_preds, nullptr, out, row_ids, n_out, flags, stream);
}

extern "C" bolt_status bolt_compact_mask(bolt_ctx* ctx, const bolt_col_view* cols, int32_t n_cols, const uint8_t* mask,
                                         bolt_col_mut* out, bolt_col_mut* row_ids, uint64_t* n_out, uint32_t flags,
                                         bolt_stream stream) {
    if (!mask) return ctx ? fail(ctx, BOLT_ERR_INVALID, "compaction: no mask") : BOLT_ERR_INVALID;
    return compact_common(ctx, cols, n_cols, nullptr, 0, mask, out, row_ids, n_out, flags, stream);
}
