// radix_sort.cu — onesweep LSD radix sort producing stable permutations for
// one or many independent segments at once.
//
// Replaces the reference's 4-bit LSD radix with a host scan per pass
// (src/exec/gpu_sort.rs:995-1230, src/jit/sort_kernel_radix.rs:489-991):
//   * one histogram kernel reads the keys once and counts all digit
//     positions of every segment (8-bit digits: 4 passes for 32-bit keys,
//     8 for 64-bit);
//   * one kernel per digit: tiles of 4096 (64-bit) or 5120 (32-bit) keys are
//     taken in arrival order from a flattened (segment, tile) list; each
//     tile's digit counts (per-warp shared atomics) are published first and
//     chained across the segment's tiles with decoupled look-back (Merrill &
//     Garland 2016); the keys are ranked per warp (stable: element order
//     within a warp's part of the tile, warps in order; the lanes holding one
//     digit find each other through a shared mask word), staged digit-sorted
//     in shared memory and written out in coalesced runs;
//   * a digit where all of a segment's keys fall in one bucket is skipped
//     for that segment on the device;
//   * the first pass applies the key transform of gpu_sort.rs:1089-1163 to
//     the raw column and generates the row-index payload; the last pass
//     writes only the payload (the permutation) to its destination.
// Many GROUP BY queries finalised together sort as many segments in the
// same handful of launches.
//
// A pass costs the same whatever its digit says about the order, and after
// the highest few digits most keys already differ from their neighbours. So
// sort_plan_kernel looks at a sample of each segment's keys and, where it
// pays, schedules passes for only the top k varying digits; sort_local_kernel
// then finishes every run of keys with equal top digits inside shared memory.
// 2^28 uniform 64-bit keys take two passes and the local step instead of
// eight passes (19.2 -> 8.4 ms: histogram 1.0, two passes 4.6, local step
// 2.7; 30M keys 2.29 -> 1.05 ms, 30M uniform 32-bit keys 0.93 -> 0.83 ms).
// A value shared by many rows is let through in a sweep (1 % of 2^28 rows:
// 19.1 -> 10.3 ms). Segments with few varying digits, or whose keys crowd
// into long runs of many values, keep the full LSD schedule.
#include "radix_sort.cuh"

#include "bulk.cuh"

#include <algorithm>

namespace bolt {
namespace {

constexpr int SORT_BLOCK = 256;
// Keys per thread in a pass: 32-bit keys leave registers and shared memory
// for larger tiles (fewer tiles to chain, more independent loads per thread).
constexpr int SORT_ITEMS_32 = 20;
constexpr int SORT_ITEMS_64 = 16;
constexpr int SORT_TILE_MIN = SORT_BLOCK * SORT_ITEMS_64;
constexpr int HIST_CHUNK = 4096;
constexpr int HIST_BLOCK = 256;
constexpr uint32_t LB_AGG = 1u << 30;
constexpr uint32_t LB_INC = 2u << 30;
constexpr uint32_t LB_VAL = (1u << 30) - 1;
constexpr uint32_t LB_SPIN_LIMIT = 1u << 22;
constexpr int LB_WINDOW = 8;  // look-back words read per round trip
constexpr int PLAN_BLOCK = 1024;
constexpr uint32_t PLAN_SAMPLES = 8192;
constexpr int PLAN_PER = PLAN_SAMPLES / PLAN_BLOCK;
constexpr int LOC_BLOCK = 512;
constexpr int LOC_NW = LOC_BLOCK / 32;
constexpr int LOC_BINS_LOG2 = 14;  // bins of the local step, counted in bytes
constexpr int LOC_WORDS = (1 << LOC_BINS_LOG2) / 4;
// Keys one bin may hold (a byte counts them): every key is compared with the
// others of its bin, so chunks with longer ones take local_crowded_sort.
constexpr uint32_t LOC_BIN_MAX = 32;
// Distinct keys up to which a crowded chunk is sorted by digits first: 256 keys
// spread over 2^16 cells meet in one in 40 % of the chunks, 362 in 63 %.
constexpr uint32_t LOC_FEW = 256;
constexpr int LOC_SER_ROUNDS = 4;  // 32-key rounds per warp and tile of the serial path

template <typename K> struct KeyTraits;
template <> struct KeyTraits<uint32_t> {
    static constexpr int NPASS = 4;
    static constexpr int ITEMS = SORT_ITEMS_32;
    static constexpr int TILE = SORT_BLOCK * ITEMS;
    static constexpr int LOC_ITEMS = 12;  // keys per thread of the local step
    // Mean run length (share of its window) up to which it is used: 32-bit
    // keys drop two passes by it and lose that to runs past the window sooner.
    static constexpr double LOC_FULL = 0.8;
    // The longest run let through: this share of the rows and half a window.
    // One CTA sorts it, 16 ns a row (64-bit keys; 7 ns for 32-bit ones, fewer
    // digits), and that is what the passes left out take for runs of 5,900,
    // 9,200, 19,000 and 50,000 rows in 1, 3, 10 and 30M (32-bit keys: 5,500,
    // 12,000 and 40,000 in 5, 20 and 60M). Near a window's length the sample's
    // estimate is off by a third either way; the passes are the safe side.
    static constexpr uint32_t LOC_RUN = 2000;
};
template <> struct KeyTraits<ull> {
    static constexpr int NPASS = 8;
    static constexpr int ITEMS = SORT_ITEMS_64;
    static constexpr int TILE = SORT_BLOCK * ITEMS;
    static constexpr int LOC_ITEMS = 10;
    static constexpr double LOC_FULL = 0.9;
    static constexpr uint32_t LOC_RUN = 600;
};

struct SegDesc {
    const void* keys;
    const uint32_t* payload_in;
    uint32_t* payload_out;
    const ull* n_dev;
    ull n;
    ull buf_off;
    uint32_t item_begin;
    uint32_t hist_begin;
    uint32_t loc_begin;
};

// A run of equal top digits longer than a window: rows [s, e) of segment sg.
struct LongRun {
    ull s, e;
    ull sg;
};

// What sort_plan_kernel decided for one segment.
struct SegPlan {
    uint32_t sched;  // digits that get a pass (bit p)
    uint32_t local;  // 1: the local step finishes the order; 0: the passes do (full LSD)
    uint32_t act;    // digits that are not constant over the segment
};

struct SortArgs {
    int32_t src;
    int32_t desc;
    int32_t indirect;
    int32_t nseg;
    const SegDesc* segs;          // nullptr for one segment: seg0 (no descriptor upload before the first launch)
    SegDesc seg0;
    const uint32_t* item_begins;  // nseg + 1; the three begins are not read for one segment
    const uint32_t* hist_begins;  // nseg + 1
    const uint32_t* loc_begins;   // nseg + 1
    void* kA;
    void* kB;
    uint32_t* pA;
    uint32_t* pB;
    uint32_t* hist;        // nseg * NPASS * 256
    uint32_t* digit_base;  // nseg * NPASS * 256
    SegPlan* plan;         // nseg
    uint32_t* lookback;    // 2 * lb_stride
    uint64_t lb_stride;    // total_items * 256
    uint32_t total_items;
    uint32_t total_hist_items;
    uint32_t total_loc_items;
    uint32_t loc_range;    // rows of one work item of the local step
    uint32_t* tile_ctr;    // NPASS + 2 (the last two: the local step's items, long runs found)
    LongRun* longs;        // in the look-back words, which the last pass is done with
    uint32_t max_longs;
    uint32_t* status;
};

// Order-preserving unsigned image of a key's raw bits: one load serves
// every source type, the transform follows (so unrolled loads stay in flight
// together).
__device__ __forceinline__ uint32_t order_key(int src, uint32_t b, int desc) {
    uint32_t k = b;
    if (src == SRC_I32) {
        k = b ^ 0x80000000u;
    } else if (src == SRC_F32) {
        const uint32_t c = canon_f32_bits(__uint_as_float(b));
        k = c ^ ((uint32_t)(((int32_t)c) >> 31) | 0x80000000u);
    }
    return desc ? ~k : k;
}
__device__ __forceinline__ ull order_key(int src, ull b, int desc) {
    ull k = b;
    if (src == SRC_I64) k = b ^ 0x8000000000000000ull;
    else if (src == SRC_F64) k = f64_order_key(__longlong_as_double((long long)b));
    return desc ? ~k : k;
}

template <typename K>
__device__ __forceinline__ K raw_key(const void* p, uint64_t r) {
    return __ldg(reinterpret_cast<const K*>(p) + r);
}

// Digit of a key at bit offset `shift` (a multiple of 8): a digit never
// straddles the two 32-bit halves of a 64-bit key, so it is taken from the
// half that holds it.
template <typename K>
__device__ __forceinline__ uint32_t digit_of(K k, int shift) {
    if constexpr (sizeof(K) == 8) {
        const uint32_t h = shift >= 32 ? (uint32_t)(k >> 32) : (uint32_t)k;
        return (h >> (shift & 31)) & 0xFFu;
    } else {
        return ((uint32_t)k >> shift) & 0xFFu;
    }
}

__device__ __forceinline__ void st_volatile_u32(uint32_t* p, uint32_t v) {
    *reinterpret_cast<volatile uint32_t*>(p) = v;
}
__device__ __forceinline__ uint32_t ld_volatile_u32(const uint32_t* p) {
    return *reinterpret_cast<const volatile uint32_t*>(p);
}

// Index of the segment owning flattened item `item` (begins is nondecreasing).
__device__ __forceinline__ int seg_of(const uint32_t* begins, int nseg, uint32_t item) {
    int lo = 0, hi = nseg;  // answer in [0, nseg)
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(begins + mid) <= item) lo = mid;
        else hi = mid;
    }
    return lo;
}

__device__ __forceinline__ const SegDesc& seg_desc(const SortArgs& a, int sg) { return a.segs ? a.segs[sg] : a.seg0; }

// Rows of a segment: the device count when given, never more than the
// segment's buffers hold (a producer that ran out of room may count past it).
__device__ __forceinline__ uint64_t seg_n(const SegDesc& d) {
    if (!d.n_dev) return d.n;
    const uint64_t n = *d.n_dev;
    return n < d.n ? n : d.n;
}

// Key i of a segment's source, transformed.
template <typename K>
__device__ __forceinline__ K source_key(const SortArgs& a, const SegDesc& d, uint64_t i) {
    return order_key(a.src, raw_key<K>(d.keys, a.indirect ? d.payload_in[i] : i), a.desc);
}

// Keys that sort_plan_kernel looks at, of a segment of n rows: as many as show
// a mean run of CAP rows in some 250 pairs (m * m from n / 8), and as show a
// run of n / LOC_RUN rows in a dozen; one a thread of its block costs no more
// than a few. Part i of m equal parts gives the sample at sample_row(i).
template <typename K>
__device__ __forceinline__ uint32_t sample_count(uint64_t n) {
    uint32_t m = 256;
    auto more = [&](uint64_t mm) { return m < PLAN_BLOCK || mm < n / 8 || (m < PLAN_SAMPLES && mm < 2 * n); };
    while (m < PLAN_SAMPLES && 4 * m <= n && more((uint64_t)m * m)) m *= 2;
    return m;
}
__device__ __forceinline__ uint32_t sample_row(uint32_t i, uint32_t step) { return i * step + __umulhi(i * 2654435761u, step); }

// Digit histograms of every segment. Bound by its shared-memory counter adds
// (one per digit and key, about 7.5 lanes per SM and cycle; four copies of
// every counter in neighbouring banks changed nothing). A CTA flushes its
// counters once per segment it meets. The rows in hand, it also leaves the
// plan's samples at the start of the segment's first key buffer: gathered by
// the plan's one CTA they cost a DRAM round trip per few hundred (5M 32-bit
// keys, 4,096 samples: plan 18.1 us, 11.7 us with them at hand).
template <typename K>
__global__ void __launch_bounds__(HIST_BLOCK) sort_hist_kernel(const __grid_constant__ SortArgs a) {
    constexpr int NP = KeyTraits<K>::NPASS;
    __shared__ uint32_t h[NP * 256];
    const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    // Clear the first look-back buffer and the pass tile counters.
    for (uint64_t i = tid; i < a.lb_stride; i += stride) a.lookback[i] = 0;
    if (blockIdx.x == 0 && threadIdx.x < NP + 2) a.tile_ctr[threadIdx.x] = 0;
    for (int i = threadIdx.x; i < NP * 256; i += blockDim.x) h[i] = 0;
    int cur = -1;
    uint32_t smp = 0, smp_step = 1;  // samples of the segment, rows of one's part
    auto flush = [&]() {
        __syncthreads();
        uint32_t* gh = a.hist + (uint64_t)cur * NP * 256;
        for (int i = threadIdx.x; i < NP * 256; i += blockDim.x) {
            const uint32_t c = h[i];
            h[i] = 0;
            if (c) atomicAdd(&gh[i], c);
        }
    };
    for (uint32_t item = blockIdx.x; item < a.total_hist_items; item += gridDim.x) {
        const int sg = seg_of(a.hist_begins, a.nseg, item);
        const bool fresh = sg != cur;
        if (fresh) {
            if (cur >= 0) flush();
            __syncthreads();
            cur = sg;
        }
        const SegDesc& d = seg_desc(a, sg);
        const uint64_t n = seg_n(d);
        if (fresh) {
            smp = n > LOC_BLOCK * KeyTraits<K>::LOC_ITEMS ? sample_count<K>(n) : 0u;
            if (smp) smp_step = (uint32_t)n / smp;  // n < 2^30
        }
        const uint64_t c0 = (uint64_t)(item - d.hist_begin) * HIST_CHUNK;
        const uint64_t c1 = c0 + HIST_CHUNK < n ? c0 + HIST_CHUNK : n;
        for (uint64_t i0 = c0 + threadIdx.x; i0 < c1; i0 += 4 * blockDim.x) {
            K raw[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint64_t i = i0 + (uint64_t)u * blockDim.x;
                raw[u] = 0;
                if (i < c1) raw[u] = raw_key<K>(d.keys, a.indirect ? d.payload_in[i] : i);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (i0 + (uint64_t)u * blockDim.x >= c1) continue;
                const K k = order_key(a.src, raw[u], a.desc);
#pragma unroll
                for (int p = 0; p < NP; ++p) atomicAdd(&h[p * 256 + digit_of<K>(k, 8 * p)], 1u);
            }
        }
        if (c0 >= n) continue;
        for (uint32_t i = (uint32_t)c0 / smp_step + threadIdx.x; i < smp && (uint64_t)i * smp_step < c1; i += blockDim.x) {
            const uint32_t r = sample_row(i, smp_step);
            if (r >= c0 && r < c1) ((K*)a.kA + d.buf_off)[i] = source_key<K>(a, d, r);
        }
    }
    if (cur >= 0) flush();
}

// Sum of v over the block (every thread gets it); red holds one word per warp.
__device__ __forceinline__ ull block_sum(ull v, ull* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    v = (threadIdx.x & 31) < (blockDim.x >> 5) ? red[threadIdx.x & 31] : 0ull;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Smallest mn and largest mx over the block, in every thread (red: two words
// per warp).
template <typename K>
__device__ __forceinline__ void block_min_max(K& mn, K& mx, ull* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const K a = __shfl_xor_sync(0xffffffffu, mn, o), b = __shfl_xor_sync(0xffffffffu, mx, o);
        mn = a < mn ? a : mn;
        mx = b > mx ? b : mx;
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 0) {
        red[2 * (threadIdx.x >> 5)] = mn;
        red[2 * (threadIdx.x >> 5) + 1] = mx;
    }
    __syncthreads();
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) {
        const K a = (K)red[2 * i], b = (K)red[2 * i + 1];
        mn = a < mn ? a : mn;
        mx = b > mx ? b : mx;
    }
}

// One CTA per segment: exclusive scan of each digit histogram (warp p: digit
// p), then the schedule.
//
// Full LSD runs a pass for every digit that is not constant over the
// segment. The short schedule runs the top k of them and leaves the rest to
// the local step, whose windows hold a few thousand keys: it needs the runs
// of keys that agree in the top k digits to be shorter than that. Their
// row-weighted mean length is n * P(two keys agree): for one digit the
// histogram says it, for more it is estimated from the agreeing pairs of a
// sample, counted in a shared hash table (2^28 uniform keys, k = 2: 512 pairs
// of 8,192 samples expected for the true 4,096); a single long run that the
// mean does not show is seen as many samples in one run. A run that is mostly
// one value (zeros, infinities, a default) counts by its other samples only:
// the local step lets the value's rows through in one sweep. All of it only
// steers the speed: the local step orders runs of any length.
struct SampleRuns {
    uint32_t pairs;     // agreeing pairs
    uint32_t longest;   // most samples in one run
    uint32_t hottest;   // most samples of one value left out of the two
};

// Counts the runs of equal key >> sh among the block's samples (cnt_s per
// thread). tab: 32-bit hashes of the prefixes, mask + 1 slots, half empty;
// cnt: samples | samples that differ from the slot's first << 16; fst: hash
// of the slot's first key. One block does this between two launches, so it is
// all latency: one CAS a sample, then counts that wait for nothing, and one
// round of reductions.
template <typename K>
__device__ __forceinline__ SampleRuns sample_runs(const K (&smp)[PLAN_PER], int cnt_s, int sh, uint32_t mask, uint32_t* tab,
                                                  uint32_t* cnt, uint32_t* fst, uint32_t* red) {
    __syncthreads();
    for (uint32_t i = 4 * threadIdx.x; i <= mask; i += 4 * PLAN_BLOCK) {
        *reinterpret_cast<uint4*>(tab + i) = make_uint4(0, 0, 0, 0);
        *reinterpret_cast<uint4*>(cnt + i) = make_uint4(0, 0, 0, 0);
    }
    __syncthreads();
    uint32_t at[PLAN_PER], own[PLAN_PER];
#pragma unroll
    for (int u = 0; u < PLAN_PER; ++u) {
        if (u >= cnt_s) continue;
        const ull hp = (ull)(smp[u] >> sh) * 0x9E3779B97F4A7C15ull;
        const uint32_t sig = (uint32_t)(hp >> 32) | 1u;
        own[u] = (uint32_t)(((ull)smp[u] * 0xD6E8FEB86659FD93ull) >> 32);
        uint32_t h = (uint32_t)(hp >> 40) & mask;
        for (uint32_t probe = 0; probe <= mask; ++probe) {
            const uint32_t old = atomicCAS(&tab[h], 0u, sig);
            if (old == 0) fst[h] = own[u];
            if (old == 0 || old == sig) break;
            h = (h + 1) & mask;
        }
        at[u] = h;
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < PLAN_PER; ++u)
        if (u < cnt_s) atomicAdd(&cnt[at[u]], fst[at[u]] == own[u] ? 1u : 0x10001u);
    __syncthreads();
    SampleRuns r{0, 0, 0};
    for (uint32_t i = threadIdx.x; i <= mask; i += PLAN_BLOCK) {
        const uint32_t all = cnt[i] & 0xFFFFu, other = cnt[i] >> 16, same = all - other;
        uint32_t c = all;
        if (same >= 4 && other * 4 <= all) {
            c = other + 1;
            r.hottest = max(r.hottest, same);
        }
        r.pairs += c * (c ? c - 1 : 0) / 2;
        r.longest = max(r.longest, c);
    }
    // (pairs fit 32 bits: 8,192 samples have 33.5M)
    r.pairs = __reduce_add_sync(0xffffffffu, r.pairs);
    r.longest = __reduce_max_sync(0xffffffffu, r.longest);
    r.hottest = __reduce_max_sync(0xffffffffu, r.hottest);
    if ((threadIdx.x & 31) == 0) {
        red[threadIdx.x >> 5] = r.pairs;
        red[32 + (threadIdx.x >> 5)] = r.longest;
        red[64 + (threadIdx.x >> 5)] = r.hottest;
    }
    __syncthreads();
    r.pairs = __reduce_add_sync(0xffffffffu, red[threadIdx.x & 31]);
    r.longest = __reduce_max_sync(0xffffffffu, red[32 + (threadIdx.x & 31)]);
    r.hottest = __reduce_max_sync(0xffffffffu, red[64 + (threadIdx.x & 31)]);
    return r;
}

template <typename K>
__global__ void __launch_bounds__(PLAN_BLOCK) sort_plan_kernel(const __grid_constant__ SortArgs a) {
    constexpr int NP = KeyTraits<K>::NPASS;
    constexpr uint32_t CAP = LOC_BLOCK * KeyTraits<K>::LOC_ITEMS;
    extern __shared__ __align__(16) unsigned char plan_sm[];
    uint32_t* tab = reinterpret_cast<uint32_t*>(plan_sm);  // 2 * PLAN_SAMPLES words
    uint32_t* cnt = tab + 2 * PLAN_SAMPLES;                // 2 * PLAN_SAMPLES words
    uint32_t* fst = cnt + 2 * PLAN_SAMPLES;                // 2 * PLAN_SAMPLES words
    __shared__ uint32_t s_act;
    static_assert(PLAN_BLOCK == 1024, "red: three words a warp, or a 64-bit one");
    __shared__ ull red[48];
    const int sg = blockIdx.x;
    const SegDesc& d = seg_desc(a, sg);
    const uint64_t n = seg_n(d);
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    if (t == 0) s_act = 0;
    const uint32_t m = sample_count<K>(n), step = (uint32_t)n / m;  // n < 2^30
    // (On their way while the histograms are scanned.)
    K smp[PLAN_PER];
    int cnt_s = 0;
    if (n > CAP) {
#pragma unroll
        for (int u = 0; u < PLAN_PER; ++u) {
            const uint32_t i = (uint32_t)u * PLAN_BLOCK + t;
            smp[u] = 0;
            if (i < m) {
                smp[u] = ((const K*)a.kA + d.buf_off)[i];
                cnt_s = u + 1;
            }
        }
    }
    __syncthreads();
    if (w < NP) {
        const uint32_t* hist = a.hist + ((uint64_t)sg * NP + w) * 256;
        uint32_t* base = a.digit_base + ((uint64_t)sg * NP + w) * 256;
        uint32_t v[8], sum = 0, big = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            v[i] = hist[lane * 8 + i];
            sum += v[i];
            big = v[i] > big ? v[i] : big;
        }
        uint32_t x = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        x -= sum;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            base[lane * 8 + i] = x;
            x += v[i];
        }
        big = __reduce_max_sync(0xffffffffu, big);
        if (lane == 0 && (uint64_t)big != n) atomicOr(&s_act, 1u << w);
    }
    __syncthreads();
    const uint32_t act = s_act;
    const int na = __popc(act);
    SegPlan plan = {act ? act : 1u, 0u, act};
    if (n <= CAP) {
        plan = {0u, 1u, act};  // one window of the local step
    } else if (na >= 3) {
        const uint64_t long_run = CAP / 2 + n / KeyTraits<K>::LOC_RUN;
        const double rows_per_pair = 2.0 * (double)n / ((double)m * (double)(m - 1));
        // The local step costs about one and a half passes.
        uint32_t sched = 0;
        for (int k = 1; k + 2 <= na; ++k) {
            const int top = 31 - __clz(act & ~sched);
            sched |= 1u << top;
            double mean;
            bool many;
            if (k == 1) {
                const uint32_t c = t < 256 ? a.hist[((uint64_t)sg * NP + top) * 256 + t] : 0u;
                mean = (double)block_sum((ull)c * c, red) / (double)n;
                many = __syncthreads_or(c > CAP + n / 2048);
            } else {
                const SampleRuns runs = sample_runs<K>(smp, cnt_s, 8 * top, 2 * m - 1, tab, cnt, fst, reinterpret_cast<uint32_t*>(red));
                mean = rows_per_pair * (double)runs.pairs;
                // (one CTA sweeps a hot value's run, 4 * CAP rows in some
                // 25 us: up to that or 1/64 of the rows)
                many = (runs.longest >= 6 && runs.longest * step > long_run) ||
                       runs.hottest * step > max((uint64_t)CAP * 4, n / 64);
            }
            if (!many && mean <= KeyTraits<K>::LOC_FULL * CAP) {
                plan = {sched, 1u, act};
                break;
            }
        }
    }
    if (t == 0) a.plan[sg] = plan;
}

template <typename K>
__global__ void __launch_bounds__(SORT_BLOCK, 3) sort_pass_kernel(const __grid_constant__ SortArgs a, int p) {
    constexpr int NW = SORT_BLOCK / 32;
    constexpr int SORT_ITEMS = KeyTraits<K>::ITEMS;
    constexpr int SORT_TILE = KeyTraits<K>::TILE;
    __shared__ uint32_t s_item;
    __shared__ uint32_t warp_pos[NW][256];  // per-warp digit counts, then each warp's next staged position
    __shared__ uint32_t peer_bits[NW][256];  // per-warp lane masks of the lanes holding a digit
    __shared__ uint32_t gdelta[256];         // global position of staged position 0, per digit
    __shared__ uint32_t wsum[NW];
    // Staged tile: keys (or, in the last pass, the digit of every position)
    // and payloads (3 CTAs of 256 threads per SM).
    extern __shared__ __align__(16) unsigned char dyn[];
    K* stage_key = reinterpret_cast<K*>(dyn);
    uint32_t* stage_pay = reinterpret_cast<uint32_t*>(dyn + sizeof(K) * SORT_TILE);
    uint8_t* stage_dig = dyn + (sizeof(K) + 4) * SORT_TILE;

    // One segment whose schedule skips this digit: nothing to do.
    if (a.nseg == 1 && !((a.plan[0].sched >> p) & 1u)) return;
    // CTAs stay and take tiles in arrival order, so a skipped pass costs one
    // small grid and not a launch per tile.
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) s_item = atomicAdd(&a.tile_ctr[p], 1u);
        for (int i = threadIdx.x; i < NW * 256; i += SORT_BLOCK) {
            (&warp_pos[0][0])[i] = 0;
            (&peer_bits[0][0])[i] = 0;
        }
        __syncthreads();
        const uint32_t item = s_item;
        if (item >= a.total_items) return;
        const int sg = seg_of(a.item_begins, a.nseg, item);
        const SegDesc& d = seg_desc(a, sg);
        const SegPlan plan = a.plan[sg];
        const uint32_t active = plan.sched;
        if (!((active >> p) & 1u)) continue;
        const uint64_t n = seg_n(d);
        const uint32_t tile = item - d.item_begin;
        if ((uint64_t)tile * SORT_TILE >= n) continue;

        const uint32_t before = active & ((1u << p) - 1u);
        const bool first = before == 0;
        const bool last = !plan.local && (active >> (p + 1)) == 0;
        const int kidx = __popc(before);
        const K* kin = ((kidx & 1) ? (const K*)a.kA : (const K*)a.kB) + d.buf_off;
        const uint32_t* pin = ((kidx & 1) ? a.pA : a.pB) + d.buf_off;
        K* kout = last ? nullptr : ((kidx & 1) ? (K*)a.kB : (K*)a.kA) + d.buf_off;
        uint32_t* pout = last ? d.payload_out : ((kidx & 1) ? a.pB : a.pA) + d.buf_off;
        uint32_t* lb = a.lookback + (uint64_t)(kidx & 1) * a.lb_stride;
        uint32_t* lb_next = a.lookback + (uint64_t)((kidx + 1) & 1) * a.lb_stride;

        const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
        uint32_t* peers_w = peer_bits[w];
        const uint64_t seg0 = (uint64_t)tile * SORT_TILE + (uint64_t)w * 32 * SORT_ITEMS;
        const int shift = 8 * p;
        const bool full = (uint64_t)(tile + 1) * SORT_TILE <= n;
        K key[SORT_ITEMS];
        uint32_t pay[SORT_ITEMS];
        if (first) {
            // Raw key bits first (all loads in flight), then the transform.
            if (a.indirect) {
#pragma unroll
                for (int j = 0; j < SORT_ITEMS; ++j) {
                    const uint64_t e = seg0 + (uint64_t)j * 32 + lane;
                    pay[j] = (full || e < n) ? d.payload_in[e] : 0u;
                }
#pragma unroll
                for (int j = 0; j < SORT_ITEMS; ++j) {
                    const uint64_t e = seg0 + (uint64_t)j * 32 + lane;
                    key[j] = (full || e < n) ? raw_key<K>(d.keys, pay[j]) : (K)0;
                }
            } else {
#pragma unroll
                for (int j = 0; j < SORT_ITEMS; ++j) {
                    const uint64_t e = seg0 + (uint64_t)j * 32 + lane;
                    key[j] = 0;
                    pay[j] = 0;
                    if (full || e < n) {
                        pay[j] = d.payload_in ? d.payload_in[e] : (uint32_t)e;
                        key[j] = raw_key<K>(d.keys, e);
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < SORT_ITEMS; ++j) key[j] = order_key(a.src, key[j], a.desc);
        } else {
#pragma unroll
            for (int j = 0; j < SORT_ITEMS; ++j) {
                const uint64_t e = seg0 + (uint64_t)j * 32 + lane;
                key[j] = 0;
                pay[j] = 0;
                if (full || e < n) {
                    key[j] = kin[e];
                    pay[j] = pin[e];
                }
            }
        }
        // Early counts: per-warp digit histograms from shared atomics, so the
        // tile's counts are published before the (longer) ranking and later
        // tiles' look-backs find them sooner.
#pragma unroll
        for (int j = 0; j < SORT_ITEMS; ++j) {
            const uint64_t e = seg0 + (uint64_t)j * 32 + lane;
            if (full || e < n) atomicAdd(&warp_pos[w][digit_of<K>(key[j], shift)], 1u);
        }
        __syncthreads();
        const uint32_t dg_me = threadIdx.x;  // SORT_BLOCK == 256: one digit per thread
        uint32_t cnt[NW];
        uint32_t run = 0;
#pragma unroll
        for (int ww = 0; ww < NW; ++ww) {
            cnt[ww] = warp_pos[ww][dg_me];
            run += cnt[ww];
        }
        st_volatile_u32(lb + (uint64_t)item * 256 + dg_me, (tile == 0 ? LB_INC : LB_AGG) | run);
        // Exclusive scan of the tile's digit counts; each warp's first staged
        // position per digit follows.
        uint32_t x = run;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) wsum[w] = x;
        __syncthreads();
        uint32_t tile_off = x - run;
        for (int i = 0; i < w; ++i) tile_off += wsum[i];
        {
            uint32_t off = tile_off;
#pragma unroll
            for (int ww = 0; ww < NW; ++ww) {
                warp_pos[ww][dg_me] = off;
                off += cnt[ww];
            }
        }
        __syncthreads();

        // Stable ranking in element order (items in order, lanes in order within
        // an item), straight to the staged position. The lanes holding the same
        // digit find each other through one shared mask word per (warp, digit);
        // the highest of them advances the warp's position for that digit.
#pragma unroll
        for (int j = 0; j < SORT_ITEMS; ++j) {
            const uint64_t e = seg0 + (uint64_t)j * 32 + lane;
            const bool valid = full || e < n;
            const uint32_t dg = digit_of<K>(key[j], shift);
            if (valid) atomicOr(&peers_w[dg], 1u << lane);
            __syncwarp();
            const uint32_t peers = valid ? peers_w[dg] : (1u << lane);
            __syncwarp();
            const int leader = 31 - __clz(peers);
            uint32_t b = 0;
            if (valid && lane == leader) {
                peers_w[dg] = 0;
                b = warp_pos[w][dg];
                warp_pos[w][dg] = b + __popc(peers);
            }
            b = __shfl_sync(0xffffffffu, b, leader);
            if (valid) {
                const uint32_t pos = b + __popc(peers & lanemask_lt());
                if (kout) stage_key[pos] = key[j];
                else stage_dig[pos] = (uint8_t)dg;  // the last pass stages no keys
                stage_pay[pos] = pay[j];
            }
            __syncwarp();
        }

        // Look back over the segment's earlier tiles, LB_WINDOW words in flight
        // at a time: sum aggregates until an inclusive prefix.
        {
            uint32_t excl = 0;
            if (tile != 0) {
                int64_t t = (int64_t)item - 1;
                const int64_t t_end = (int64_t)d.item_begin;
                uint32_t spins = 0;
                while (t >= t_end) {
                    const int cnt_w = (t - t_end + 1) < LB_WINDOW ? (int)(t - t_end + 1) : LB_WINDOW;
                    uint32_t v[LB_WINDOW];
#pragma unroll
                    for (int i = 0; i < LB_WINDOW; ++i)
                        v[i] = i < cnt_w ? ld_volatile_u32(lb + (uint64_t)(t - i) * 256 + dg_me) : 0u;
                    int used = 0;
                    bool done = false, stalled = false;
#pragma unroll
                    for (int i = 0; i < LB_WINDOW; ++i) {
                        if (done || stalled || i >= cnt_w) continue;
                        const uint32_t st = v[i] >> 30;
                        if (st == 0) {
                            stalled = true;  // not published yet: poll again from here
                            continue;
                        }
                        excl += v[i] & LB_VAL;
                        ++used;
                        if (st == 2) done = true;
                    }
                    if (done) break;
                    t -= used;
                    if (stalled) {
                        if (++spins > LB_SPIN_LIMIT) {
                            atomicOr(a.status, ST_FLAG_TIMEOUT);
                            break;
                        }
                        if (spins > 4) __nanosleep(64);
                    }
                }
                st_volatile_u32(lb + (uint64_t)item * 256 + dg_me, LB_INC | ((excl + run) & LB_VAL));
            }
            lb_next[(uint64_t)item * 256 + dg_me] = 0;
            // Positions fit in 32 bits (n < 2^30), so the difference wraps safely.
            gdelta[dg_me] = a.digit_base[((uint64_t)sg * KeyTraits<K>::NPASS + p) * 256 + dg_me] + excl - tile_off;
        }
        __syncthreads();

        // Coalesced runs out of the staged tile.
        const uint64_t tb = (uint64_t)tile * SORT_TILE;
        const uint32_t tile_n = (uint32_t)((n - tb) < (uint64_t)SORT_TILE ? (n - tb) : (uint64_t)SORT_TILE);
        const uint32_t n32 = (uint32_t)n;  // n < 2^30
        if (kout) {
            for (uint32_t i = threadIdx.x; i < tile_n; i += SORT_BLOCK) {
                const K k = stage_key[i];
                const uint32_t g = gdelta[digit_of<K>(k, shift)] + i;
                if (g >= n32) {  // only reachable after a look-back timeout
                    atomicOr(a.status, ST_FLAG_TIMEOUT);
                    continue;
                }
                kout[g] = k;
                pout[g] = stage_pay[i];
            }
        } else {
            for (uint32_t i = threadIdx.x; i < tile_n; i += SORT_BLOCK) {
                const uint32_t g = gdelta[stage_dig[i]] + i;
                if (g >= n32) {
                    atomicOr(a.status, ST_FLAG_TIMEOUT);
                    continue;
                }
                pout[g] = stage_pay[i];
            }
        }
    }
}

// First position >= p of the rows [0, n) whose prefix (key >> sh) differs from
// its predecessor's (0 and n count as such positions). The prefixes are
// nondecreasing, so 32 lanes narrow the range 32-fold per round trip, from a
// first guess of one work item's length. Whole warp.
template <typename K>
__device__ __forceinline__ uint64_t run_start_from(const K* keys, uint64_t p, uint64_t n, int sh) {
    if (p == 0 || p >= n) return p < n ? p : n;
    const uint32_t lane = threadIdx.x & 31;
    const K pre = keys[p - 1] >> sh;
    uint64_t lo = p, hi = n;  // the answer is in [lo, hi]
    uint64_t step = 256;
    while (lo < hi) {
        // Lane l probes lo + l * step.
        const uint64_t at = lo + lane * step;
        const bool past = at >= hi || (keys[at] >> sh) != pre;
        const uint32_t m = __ballot_sync(0xffffffffu, past);
        if (m == 0) {  // beyond the last probe
            lo = lo + 31 * step + 1;
            step = (hi - lo + 31) / 32;
            if (step == 0) step = 1;
            continue;
        }
        const int f = __ffs(m) - 1;
        const uint64_t fa = lo + f * step;
        hi = fa < hi ? fa : hi;
        if (f == 0) return hi;
        lo = lo + (f - 1) * step + 1;
        step = (hi - lo + 31) / 32;
        if (step == 0) step = 1;
    }
    return hi;
}

// Stable LSD radix sort of len rows (keys kx, payloads px) by one CTA, tile
// after tile, over the digits that vary among them; the sorted payloads go to
// `out`, those from gap_at on `gap` places further. For the rare runs longer
// than a window. It orders row numbers, in ix and iy (len words each), and
// leaves the rows where they are. cnt: LOC_NW * 256 words; base: 256 words.
template <typename K>
__device__ __forceinline__ void local_serial_sort(const K* kx, const uint32_t* px, uint32_t* ix, uint32_t* iy, uint64_t len,
                                               uint32_t* out, uint64_t gap_at, uint64_t gap, uint32_t* cnt, uint32_t* base,
                                               ull* red) {
    constexpr int NP = KeyTraits<K>::NPASS;
    const int t = threadIdx.x, w = t >> 5, lane = t & 31;
    bool first = true;  // the order so far is the identity
    ull vary = 0;
    const K k0 = kx[0];
    for (uint64_t i = t; i < len; i += LOC_BLOCK) vary |= (ull)(kx[i] ^ k0);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) vary |= __shfl_xor_sync(0xffffffffu, vary, o);
    __syncthreads();
    if (lane == 0) red[w] = vary;
    __syncthreads();
    for (int i = 0; i < LOC_NW; ++i) vary |= red[i];
    for (int p = 0; p < NP; ++p) {
        if (((vary >> (8 * p)) & 0xFFull) == 0) continue;
        const int sh = 8 * p;
        if (t < 256) base[t] = 0;
        __syncthreads();
        for (uint64_t i = t; i < len; i += LOC_BLOCK) atomicAdd(&base[digit_of<K>(kx[i], sh)], 1u);
        __syncthreads();
        if (w == 0) {  // exclusive scan of the 256 counts
            uint32_t v[8], sum = 0;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                v[i] = base[lane * 8 + i];
                sum += v[i];
            }
            uint32_t x = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            x -= sum;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                base[lane * 8 + i] = x;
                x += v[i];
            }
        }
        for (uint64_t t0 = 0; t0 < len; t0 += LOC_BLOCK * LOC_SER_ROUNDS) {
            for (int i = t; i < LOC_NW * 256; i += LOC_BLOCK) cnt[i] = 0;
            __syncthreads();
            const uint64_t w0 = t0 + (uint64_t)w * 32 * LOC_SER_ROUNDS + lane;
#pragma unroll
            for (int r = 0; r < LOC_SER_ROUNDS; ++r) {
                const uint64_t i = w0 + 32 * r;
                if (i < len) atomicAdd(&cnt[w * 256 + digit_of<K>(kx[first ? (uint32_t)i : ix[i]], sh)], 1u);
            }
            __syncthreads();
            if (t < 256) {
                uint32_t off = base[t];
                for (int ww = 0; ww < LOC_NW; ++ww) {
                    const uint32_t c = cnt[ww * 256 + t];
                    cnt[ww * 256 + t] = off;
                    off += c;
                }
                base[t] = off;
            }
            __syncthreads();
            for (int r = 0; r < LOC_SER_ROUNDS; ++r) {
                const uint64_t i = w0 + 32 * r;
                const bool in = i < len;
                const uint32_t on = __ballot_sync(0xffffffffu, in);
                if (in) {
                    const uint32_t id = first ? (uint32_t)i : ix[i];
                    const uint32_t dg = digit_of<K>(kx[id], sh);
                    const uint32_t peers = __match_any_sync(on, dg);
                    const uint32_t b = cnt[w * 256 + dg];
                    __syncwarp(on);
                    if (lane == 31 - __clz(peers)) cnt[w * 256 + dg] = b + __popc(peers);
                    iy[b + __popc(peers & lanemask_lt())] = id;
                }
                __syncwarp();
            }
            __syncthreads();
        }
        uint32_t* const it = ix;
        ix = iy;
        iy = it;
        first = false;
    }
    for (uint64_t i = t; i < len; i += LOC_BLOCK) out[i + (i >= gap_at ? gap : 0)] = px[first ? (uint32_t)i : ix[i]];
    __syncthreads();
}

// The bytes of a key with the digits that vary over the segment packed at the
// bottom, in order, and the constant ones above them: the same order between
// keys of the segment, with no constant bits in between.
struct Packer {
    uint32_t lo, hi;
    __device__ __forceinline__ Packer(uint32_t act, int nbytes) {
        ull sel = 0;
        int at = 0;
        for (int pass = 0; pass < 2; ++pass)
            for (int b = 0; b < nbytes; ++b)
                if ((((act >> b) & 1u) != 0) == (pass == 0)) sel |= (ull)b << (4 * at++);
        lo = (uint32_t)sel & 0xFFFFu;
        hi = (uint32_t)(sel >> 16) & 0xFFFFu;
    }
    __device__ __forceinline__ ull operator()(ull k) const {
        const uint32_t x = (uint32_t)k, y = (uint32_t)(k >> 32);
        return ((ull)__byte_perm(x, y, hi) << 32) | __byte_perm(x, y, lo);
    }
    __device__ __forceinline__ uint32_t operator()(uint32_t k) const { return __byte_perm(k, 0u, lo); }
};

// One stable counting pass of the crowded-chunk sort over the row numbers
// src -> dst (identity: src is 0, 1, 2, ...), by digit(row).
template <int ITEMS, class Digit>
__device__ __forceinline__ void local_pass(const uint16_t* src, uint16_t* dst, bool identity, uint32_t len, uint32_t* cnt,
                                           uint32_t* wsum, Digit digit) {
    const int t = threadIdx.x, w = t >> 5, lane = t & 31;
    for (int i = t; i < LOC_NW * 256; i += LOC_BLOCK) cnt[i] = 0;
    __syncthreads();
    uint32_t rd[ITEMS];  // row | digit << 16
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        const uint32_t p = (uint32_t)(w * ITEMS + r) * 32 + lane;
        rd[r] = 0;
        if (p < len) {
            const uint32_t id = identity ? p : src[p], dg = digit(id);
            rd[r] = id | (dg << 16);
            atomicAdd(&cnt[w * 256 + dg], 1u);
        }
    }
    __syncthreads();
    uint32_t run = 0, x = 0;
    if (t < 256) {
        for (int ww = 0; ww < LOC_NW; ++ww) run += cnt[ww * 256 + t];
        x = run;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) wsum[w] = x;
    }
    __syncthreads();
    if (t < 256) {
        uint32_t off = x - run;
        for (int i = 0; i < w; ++i) off += wsum[i];
        for (int ww = 0; ww < LOC_NW; ++ww) {
            const uint32_t c = cnt[ww * 256 + t];
            cnt[ww * 256 + t] = off;
            off += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        const uint32_t p = (uint32_t)(w * ITEMS + r) * 32 + lane;
        const bool in = p < len;
        const uint32_t dg = rd[r] >> 16;
        uint32_t peers = __ballot_sync(0xffffffffu, in);
#pragma unroll
        for (int bit = 0; bit < 8; ++bit) {
            const uint32_t on = (dg >> bit) & 1u;
            const uint32_t bal = __ballot_sync(0xffffffffu, on);
            peers &= on ? bal : ~bal;
        }
        uint32_t b = 0;
        if (in) b = cnt[w * 256 + dg];
        __syncwarp();
        if (in) {
            if (lane == 31 - __clz(peers)) cnt[w * 256 + dg] = b + __popc(peers);
            dst[b + __popc(peers & lanemask_lt())] = (uint16_t)(rd[r] & 0xFFFFu);
        }
        __syncwarp();
    }
    __syncthreads();
}

// Sorts a chunk whose keys crowd into too few bins (repeated keys, or gaps
// between clusters), in shared memory: skey holds its keys in chunk order,
// spay the payloads; payloads from gap_at on go `gap` places further. Row
// numbers (ia, ib) are sorted. A few keys that repeat (digits) are settled by
// two stable counting passes over the leading 16 bits of the keys' range;
// where those do not leave the rows in order, and for many keys straight away,
// a stable merge sort does it: each thread sorts LOC_ITEMS neighbours in
// registers, then pairs of lists are merged, each thread its own LOC_ITEMS
// outputs of a pair from where a binary search says they begin; lists in order
// are only copied, as most are once they are longer than the runs. (With two
// CTAs per SM at it, the counting passes take 26 us a chunk, the merge sort
// 40-50: 10M prices of 100,000 values 610 us, by merging alone 760. Where the
// passes do not settle it, up to eight more took 53 us: 5M floats with 0.4 %
// special values 313 us, by merging alone 278, every digit in a pass 280.)
template <typename K>
__device__ __noinline__ void local_crowded_sort(const K* skey, const uint32_t* spay, uint16_t* ia, uint16_t* ib, uint32_t len,
                                                bool digits, uint32_t act, K lo, int bits, uint32_t* out, uint32_t gap_at,
                                                uint64_t gap, uint32_t* cnt, uint32_t* wsum) {
    constexpr uint32_t ITEMS = KeyTraits<K>::LOC_ITEMS;
    const uint32_t t = threadIdx.x;
    if (digits) {
        const Packer pack(act, (int)sizeof(K));
        const int top = bits > 16 ? bits - 16 : 0;
        local_pass<ITEMS>(ia, ia, true, len, cnt, wsum, [&](uint32_t i) { return (uint32_t)((K)(pack(skey[i]) - lo) >> top) & 0xFFu; });
        local_pass<ITEMS>(ia, ib, false, len, cnt, wsum,
                          [&](uint32_t i) { return (uint32_t)((K)(pack(skey[i]) - lo) >> top >> 8) & 0xFFu; });
        bool ok = true;
        if (bits > 16)
            for (uint32_t p = t + 1; p < len; p += LOC_BLOCK) ok = ok && skey[ib[p - 1]] <= skey[ib[p]];
        if (__syncthreads_and(ok)) {
            for (uint32_t p = t; p < len; p += LOC_BLOCK) out[p + (p >= gap_at ? gap : 0)] = spay[ib[p]];
            __syncthreads();
            return;
        }
    }
    {
        K k[ITEMS];
        uint32_t id[ITEMS];
#pragma unroll
        for (uint32_t j = 0; j < ITEMS; ++j) {
            const bool in = t * ITEMS + j < len;
            id[j] = !in ? 0u : digits ? ib[t * ITEMS + j] : t * ITEMS + j;
            k[j] = in ? skey[id[j]] : ~(K)0;  // (rows past the end stay behind equal keys)
        }
#pragma unroll
        for (uint32_t r = 0; r < ITEMS; ++r) {  // odd-even transposition: neighbours only, so it is stable
#pragma unroll
            for (uint32_t j = r & 1; j + 1 < ITEMS; j += 2) {
                const bool sw = k[j] > k[j + 1];
                const K a = sw ? k[j + 1] : k[j], b = sw ? k[j] : k[j + 1];
                const uint32_t x = sw ? id[j + 1] : id[j], y = sw ? id[j] : id[j + 1];
                k[j] = a;
                k[j + 1] = b;
                id[j] = x;
                id[j + 1] = y;
            }
        }
#pragma unroll
        for (uint32_t j = 0; j < ITEMS; ++j)
            if (t * ITEMS + j < len) ia[t * ITEMS + j] = (uint16_t)id[j];
    }
    __syncthreads();
    uint16_t *src = ia, *dst = ib;
    for (uint32_t w = ITEMS; w < len; w *= 2) {
        // Lists a (na rows) and b (nb rows) of the thread's pair; its outputs
        // are [d, d + ITEMS) of the merged list.
        const uint32_t per = 2 * w / ITEMS, base = (t / per) * 2 * w, d = (t & (per - 1)) * ITEMS;
        const uint32_t mid = min(base + w, len), end = min(base + 2 * w, len);
        if (base + d < len) {
            const uint16_t *a = src + base, *b = src + mid;
            const uint32_t na = mid - base, nb = end - mid;
            const uint32_t stop = min(d + ITEMS, na + nb);
            if (nb == 0 || skey[a[na - 1]] <= skey[b[0]]) {
                // In order already (a chunk's runs are, and equal keys):
                // the two lists, one after the other.
                for (uint32_t o = d; o < stop; ++o) dst[base + o] = a[o];
            } else {
                uint32_t lo = d > nb ? d - nb : 0, hi = min(d, na);
                while (lo < hi) {  // rows of a before output d (a's come first among equal keys)
                    const uint32_t m = (lo + hi) / 2;
                    if (skey[a[m]] <= skey[b[d - 1 - m]]) lo = m + 1;
                    else hi = m;
                }
                uint32_t i = lo, j = d - lo;
                uint32_t x = i < na ? a[i] : 0, y = j < nb ? b[j] : 0;
                K kx = skey[x], ky = skey[y];
                for (uint32_t o = d; o < stop; ++o) {
                    const bool from_a = j >= nb || (i < na && kx <= ky);
                    dst[base + o] = (uint16_t)(from_a ? x : y);
                    if (from_a) {
                        if (++i < na) kx = skey[x = a[i]];
                    } else {
                        if (++j < nb) ky = skey[y = b[j]];
                    }
                }
            }
        }
        __syncthreads();
        uint16_t* const z = src;
        src = dst;
        dst = z;
    }
    for (uint32_t p = t; p < len; p += LOC_BLOCK) out[p + (p >= gap_at ? gap : 0)] = spay[src[p]];
    __syncthreads();
}

// A run longer than a window (len rows at kin / pin) in which one value is
// frequent: a sweep counts the rows below and equal to it, a second one writes
// the equal rows' payloads in place and collects the others, in order, to be
// sorted around the gap: at skey / spay by local_crowded_sort where they fit a
// window, else in the run's part of the other buffer (kalt / palt) by
// local_serial_sort, with the run's own part, read for the last time, for its
// row numbers. So a run costs two sweeps and the sort of its other rows,
// however often its frequent value occurs (2^28 hashes with 1 % zeros and
// 20,000 ids beside them: 39.0 ms with the whole run in local_serial_sort,
// 10.9 ms). False (nothing written) when no
// value is a quarter of a sample.
template <typename K>
__device__ __forceinline__ bool local_hot_run(K* kin, uint32_t* pin, K* kalt, uint32_t* palt, uint64_t len, uint32_t cap,
                                           K* skey, uint32_t* spay, uint16_t* ia, uint32_t* out, uint32_t* cnt,
                                           uint32_t* base, uint32_t* wsum, ull* red) {
    constexpr int U = 8;
    const int t = threadIdx.x, w = t >> 5, lane = t & 31;
    // Candidate: the most frequent of 32 samples (every warp finds the same).
    const K mine = kin[(len / 32) * (uint32_t)lane + len / 64];
    const uint32_t same = (uint32_t)__popc(__match_any_sync(0xffffffffu, mine));
    const uint32_t best = __reduce_max_sync(0xffffffffu, same);
    if (best < 8) return false;
    const K hot = __shfl_sync(0xffffffffu, mine, __ffs(__ballot_sync(0xffffffffu, same == best)) - 1);
    ull below = 0, equal = 0;
    for (uint64_t i0 = t; i0 < len; i0 += LOC_BLOCK * U) {
        K k[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint64_t i = i0 + (uint64_t)u * LOC_BLOCK;
            k[u] = i < len ? kin[i] : ~(K)0;
            if (i < len) {
                below += k[u] < hot;
                equal += k[u] == hot;
            }
        }
    }
    below = block_sum(below, red);
    equal = block_sum(equal, red);
    const uint64_t n_rest = len - equal;
    const bool fits = n_rest <= cap;
    K* const krest = fits ? skey : kalt;
    uint32_t* const prest = fits ? spay : palt;
    uint64_t rest = 0;  // rows of other values before the tile
    for (uint64_t t0 = 0; t0 < len; t0 += LOC_BLOCK * U) {
        // Warp w's part: rows t0 + w * 32 * U + [0, 32 * U), 32 at a time.
        K k[U];
        uint32_t pay[U], me[U], c = 0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint64_t i = t0 + (uint64_t)(w * U + u) * 32 + lane;
            k[u] = i < len ? kin[i] : hot;
            pay[u] = i < len ? pin[i] : 0u;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            me[u] = __ballot_sync(0xffffffffu, k[u] != hot);
            c += __popc(me[u]);
        }
        __syncthreads();
        if (lane == 0) wsum[w] = c;
        __syncthreads();
        const uint32_t v = lane < LOC_NW ? wsum[lane] : 0u;
        uint32_t before = __reduce_add_sync(0xffffffffu, lane < w ? v : 0u);  // others in the earlier warps' parts
        const uint32_t all = __reduce_add_sync(0xffffffffu, v);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint64_t i = t0 + (uint64_t)(w * U + u) * 32 + lane;
            if (i < len) {
                const uint64_t others = rest + before + __popc(me[u] & lanemask_lt());
                if ((me[u] >> lane) & 1u) {
                    krest[others] = k[u];
                    prest[others] = pay[u];
                } else {
                    out[below + (i - others)] = pay[u];
                }
            }
            before += __popc(me[u]);
        }
        rest += all;
    }
    __syncthreads();
    if (fits)
        local_crowded_sort<K>(skey, spay, ia, ia + cap, (uint32_t)n_rest, false, 0u, (K)0, 0, out, (uint32_t)below, equal, cnt, wsum);
    else
        local_serial_sort<K>(kalt, palt, reinterpret_cast<uint32_t*>(kin), pin, n_rest, out, below, equal, cnt, base, red);
    return true;
}

// The runs longer than a window, one CTA each.
template <typename K>
__global__ void __launch_bounds__(LOC_BLOCK) sort_long_kernel(const __grid_constant__ SortArgs a) {
    constexpr uint32_t CAP = LOC_BLOCK * KeyTraits<K>::LOC_ITEMS;
    extern __shared__ __align__(16) unsigned char loc_sm[];
    __shared__ uint32_t s_base[256], s_wsum[LOC_NW];
    __shared__ ull red[2 * LOC_NW];
    K* skey = reinterpret_cast<K*>(loc_sm);
    uint32_t* bins = reinterpret_cast<uint32_t*>(skey + CAP);
    uint32_t* spay = bins + LOC_WORDS;
    uint16_t* ia = reinterpret_cast<uint16_t*>(spay + CAP);
    const uint32_t runs = min(a.tile_ctr[KeyTraits<K>::NPASS + 1], a.max_longs);
    for (uint32_t r = blockIdx.x; r < runs; r += gridDim.x) {
        const LongRun run = a.longs[r];
        const SegDesc& d = seg_desc(a, (int)run.sg);
        const SegPlan plan = a.plan[run.sg];
        const bool in_a = (__popc(plan.sched) & 1) != 0;
        const uint64_t at = d.buf_off + run.s, len = run.e - run.s;
        K* kin = (K*)(in_a ? a.kA : a.kB) + at;
        K* kalt = (K*)(in_a ? a.kB : a.kA) + at;
        uint32_t* pin = (in_a ? a.pA : a.pB) + at;
        uint32_t* palt = (in_a ? a.pB : a.pA) + at;
        uint32_t* out = d.payload_out + run.s;
        if (!local_hot_run<K>(kin, pin, kalt, palt, len, CAP, skey, spay, ia, out, bins, s_base, s_wsum, red))
            local_serial_sort<K>(kin, pin, reinterpret_cast<uint32_t*>(kalt), palt, len, out, len, 0, bins, s_base, red);
        __syncthreads();
    }
}

// The local step: rows sorted by their top digits (key >> sh, the "prefix")
// get their final order. A work item is loc_range rows of a segment, widened
// to whole runs of equal prefixes; the CTA walks it in chunks of whole runs,
// at most CAP rows. In a chunk every key goes to one of 16,384 bins by the
// leading bits in which the chunk's keys can differ (a monotone map, a third
// to a half of a key per bin), and is ranked against the other keys of its
// bin by (key, position in the chunk), which makes the order exact and stable
// whatever order the bin was filled in. The lanes of a warp wait for the
// longest of their 32 bins, so bins are many and short: four byte counters to
// a word, and one offset per word. Only shared-memory work per key: one
// counter add, one staged key, a compare or two, one staged payload; reads
// 12 B and writes 4 B per row.
template <typename K>
__global__ void __launch_bounds__(LOC_BLOCK, 2) sort_local_kernel(const __grid_constant__ SortArgs a) {
    constexpr int ITEMS = KeyTraits<K>::LOC_ITEMS;
    constexpr uint32_t CAP = LOC_BLOCK * ITEMS;
    extern __shared__ __align__(16) unsigned char loc_sm[];
    K* skey = reinterpret_cast<K*>(loc_sm);
    uint32_t* bins = reinterpret_cast<uint32_t*>(skey + CAP);  // LOC_WORDS: four bin counts each
    uint32_t* spay = bins + LOC_WORDS;                         // payloads in chunk order
    uint32_t* smeta = spay + CAP;                              // binned: position in the chunk, bin's length << 16, arrival << 24
    uint16_t* woff = reinterpret_cast<uint16_t*>(smeta + CAP);  // LOC_WORDS: keys before each word's bins
    __shared__ uint32_t s_item, s_heavy, s_used, s_last;
    __shared__ uint64_t s_lim[2];
    __shared__ uint32_t s_wsum[LOC_NW];
    __shared__ ull red[2 * LOC_NW];
    const int t = threadIdx.x, w = t >> 5, lane = t & 31;
    if (a.nseg == 1 && !a.plan[0].local) return;
    for (;;) {
        __syncthreads();
        if (t == 0) s_item = atomicAdd(&a.tile_ctr[KeyTraits<K>::NPASS], 1u);
        __syncthreads();
        if (s_item >= a.total_loc_items) return;
        // Infinities and NaNs, the likeliest crowded chunks, go first: their
        // longer sort is then not what the grid ends with.
        const uint32_t item = a.desc ? s_item : a.total_loc_items - 1 - s_item;
        const int sg = seg_of(a.loc_begins, a.nseg, item);
        const SegDesc& d = seg_desc(a, sg);
        const SegPlan plan = a.plan[sg];
        if (!plan.local) continue;
        const uint64_t n = seg_n(d);
        const uint64_t r0 = (uint64_t)(item - d.loc_begin) * a.loc_range;
        if (r0 >= n) continue;
        K* kA = (K*)a.kA + d.buf_off;
        K* kB = (K*)a.kB + d.buf_off;
        uint32_t* pA = a.pA + d.buf_off;
        uint32_t* pB = a.pB + d.buf_off;
        // Pass i (from 0) writes A when i is even.
        const bool in_a = (__popc(plan.sched) & 1) != 0;
        const K* kin = in_a ? kA : kB;
        const uint32_t* pin = in_a ? pA : pB;
        const bool raw = plan.sched == 0;  // no pass ran: the source itself, one chunk (n <= CAP)
        const int sh = raw ? 0 : 8 * (__ffs(plan.sched) - 1);
        const Packer pack(plan.act, (int)sizeof(K));
        const int psh = 8 * (__popc(plan.act) - __popc(plan.sched));  // the same shift on packed keys
        if (!raw && w < 2) {
            const uint64_t at = run_start_from<K>(kin, w == 0 ? r0 : min(r0 + (uint64_t)a.loc_range, n), n, sh);
            if (lane == 0) s_lim[w] = at;
        }
        __syncthreads();
        uint64_t pos = raw ? 0 : s_lim[0];
        const uint64_t end = raw ? n : s_lim[1];
        if (raw && r0 != 0) continue;
        while (pos < end) {
            const uint32_t win = end - pos < CAP ? (uint32_t)(end - pos) : CAP;
            K key[ITEMS];
#pragma unroll
            for (int j = 0; j < ITEMS; ++j) {
                const uint32_t i = (uint32_t)j * LOC_BLOCK + t;
                key[j] = 0;
                if (i < win) key[j] = raw ? source_key<K>(a, d, i) : kin[pos + i];
            }
#pragma unroll
            for (int j = 0; j < ITEMS; ++j) {
                const uint32_t i = (uint32_t)j * LOC_BLOCK + t;
                if (i < win) spay[i] = !raw ? pin[pos + i] : d.payload_in ? d.payload_in[i] : i;
            }
            // The next window on its way to L2 meanwhile.
            if (t == 0 && end - pos > win) {
                // (whole groups of 8 rows of the buffers, which start on
                // 256-byte boundaries: 16-byte aligned addresses and sizes)
                const uint64_t next = pos + win, stop = end - next < CAP ? end : next + CAP;
                const uint64_t b0 = (d.buf_off + next) & ~7ull, b1 = (d.buf_off + stop) & ~7ull;
                if (b0 < b1) {
                    bulk_prefetch_l2((const K*)(in_a ? a.kA : a.kB) + b0, (uint32_t)(b1 - b0) * (uint32_t)sizeof(K));
                    bulk_prefetch_l2((in_a ? a.pA : a.pB) + b0, (uint32_t)(b1 - b0) * 4u);
                }
            }
            // The chunk: the window up to its last run start, or all of it
            // when a run ends with it.
            uint32_t len = win;
            K kfirst = 0, klast = ~(K)0;
            if (!raw) {
                kfirst = kin[pos];
                klast = kin[pos + win - 1];
                if (pos + win < end && (kin[pos + win] >> sh) == (klast >> sh)) {
                    if (t == 0) s_last = win;
                    __syncthreads();
#pragma unroll
                    for (int j = 0; j < ITEMS; ++j) {
                        const uint32_t i = (uint32_t)j * LOC_BLOCK + t;
                        const uint32_t m = __ballot_sync(0xffffffffu, i < win && (key[j] >> sh) == (klast >> sh));
                        if (m && lane == 0) atomicMin(&s_last, i + (uint32_t)__ffs(m) - 1);
                    }
                    __syncthreads();
                    len = s_last;
                    if (len) klast = kin[pos + len - 1];
                }
            }
            if (len == 0) {  // one run longer than the window
                // (sort_long_kernel orders it: its code would cost this
                // kernel's main path registers)
                if (w == 0) {
                    const uint64_t at = run_start_from<K>(kin, pos + win, n, sh);
                    if (lane == 0) {
                        s_lim[0] = at;
                        const uint32_t q = atomicAdd(&a.tile_ctr[KeyTraits<K>::NPASS + 1], 1u);
                        if (q < a.max_longs) a.longs[q] = LongRun{pos, at, (ull)sg};
                        else atomicOr(a.status, ST_FLAG_TIMEOUT);  // only reachable after a look-back timeout
                    }
                }
                __syncthreads();
                const uint64_t e = s_lim[0];
                pos = e;
                continue;
            }
            // Bins: the leading bits of the packed key's distance from the
            // lowest one the chunk can hold.
            K lo, span;
            if (raw) {
                K mn = ~(K)0, mx = 0;
#pragma unroll
                for (int j = 0; j < ITEMS; ++j) {
                    if ((uint32_t)j * LOC_BLOCK + t < len) {
                        const K q = pack(key[j]);
                        mn = q < mn ? q : mn;
                        mx = q > mx ? q : mx;
                    }
                }
                block_min_max(mn, mx, red);
                lo = mn;
                span = mx - mn;
            } else {
                const K p0 = pack(kfirst) >> psh;
                lo = p0 << psh;
                span = (((pack(klast) >> psh) - p0) << psh) | (((K)1 << psh) - 1);
            }
            const int bits = sizeof(K) == 8 ? 64 - __clzll((ll)span) : 32 - __clz((int)span);
            const int bsh = bits > LOC_BINS_LOG2 ? bits - LOC_BINS_LOG2 : 0;
            for (int i = t; i < LOC_WORDS / 4; i += LOC_BLOCK) reinterpret_cast<uint4*>(bins)[i] = make_uint4(0, 0, 0, 0);
            if (t == 0) s_heavy = s_used = 0;
            __syncthreads();
            uint32_t br[ITEMS];  // bin | arrival number in the bin << 16
            bool heavy = false;
#pragma unroll
            for (int j = 0; j < ITEMS; ++j) {
                br[j] = 0;
                if ((uint32_t)j * LOC_BLOCK + t < len) {
                    const uint32_t b = min((uint32_t)((K)(pack(key[j]) - lo) >> bsh), (1u << LOC_BINS_LOG2) - 1);
                    const uint32_t sub = 8 * (b & 3);
                    const uint32_t r = (atomicAdd(&bins[b >> 2], 1u << sub) >> sub) & 0xFFu;
                    heavy |= r >= LOC_BIN_MAX;
                    br[j] = b | (r << 16);
                }
            }
            if (heavy) s_heavy = 1;
            __syncthreads();
            if (s_heavy) {
                // Distinct keys: flags by hash, in woff's 8,192 bytes.
                uint4* flags = reinterpret_cast<uint4*>(woff);
                static_assert(LOC_WORDS * 2 == LOC_BLOCK * 16, "one uint4 of flags a thread");
                flags[t] = make_uint4(0, 0, 0, 0);
                __syncthreads();
#pragma unroll
                for (int j = 0; j < ITEMS; ++j) {
                    const uint32_t i = (uint32_t)j * LOC_BLOCK + t;
                    if (i >= len) continue;
                    skey[i] = key[j];
                    reinterpret_cast<uint8_t*>(woff)[((ull)key[j] * 0x9E3779B97F4A7C15ull) >> 51] = 1;
                }
                __syncthreads();
                const uint4 q = flags[t];
                const uint32_t used = __reduce_add_sync(0xffffffffu, __popc(q.x) + __popc(q.y) + __popc(q.z) + __popc(q.w));
                if (lane == 0) atomicAdd(&s_used, used);
                __syncthreads();
                uint16_t* ia = reinterpret_cast<uint16_t*>(smeta);
                local_crowded_sort<K>(skey, spay, ia, ia + CAP, len, s_used > 1 && s_used <= LOC_FEW, plan.act, lo, bits, d.payload_out + pos,
                                      len, 0, bins, s_wsum);
                pos += len;
                continue;
            }
            // Exclusive scan of the words' counts, LOC_WORDS / LOC_BLOCK per thread.
            {
                constexpr int PER = LOC_WORDS / LOC_BLOCK;
                uint32_t v[PER], sum = 0;
#pragma unroll
                for (int i = 0; i < PER; i += 4) {
                    const uint4 q = *reinterpret_cast<const uint4*>(bins + t * PER + i);
                    v[i] = __dp4a(q.x, 0x01010101u, 0u);
                    v[i + 1] = __dp4a(q.y, 0x01010101u, 0u);
                    v[i + 2] = __dp4a(q.z, 0x01010101u, 0u);
                    v[i + 3] = __dp4a(q.w, 0x01010101u, 0u);
                }
#pragma unroll
                for (int i = 0; i < PER; ++i) sum += v[i];
                uint32_t x = sum;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                    if (lane >= o) x += y;
                }
                if (lane == 31) s_wsum[w] = x;
                __syncthreads();
                x -= sum;
                x += __reduce_add_sync(0xffffffffu, lane < w ? s_wsum[lane] : 0u);
#pragma unroll
                for (int i = 0; i < PER; i += 2) {
                    const uint32_t y = x + v[i];
                    *reinterpret_cast<uint32_t*>(woff + t * PER + i) = x | (y << 16);
                    x = y + v[i + 1];
                }
            }
            __syncthreads();
#pragma unroll
            for (int j = 0; j < ITEMS; ++j) {
                const uint32_t i = (uint32_t)j * LOC_BLOCK + t;
                if (i < len) {
                    const uint32_t b = br[j] & 0xFFFFu, c4 = bins[b >> 2], sub = 8 * (b & 3);
                    const uint32_t at = woff[b >> 2] + __dp4a(c4 & ((1u << sub) - 1u), 0x01010101u, 0u) + (br[j] >> 16);
                    skey[at] = key[j];
                    smeta[at] = i | (((c4 >> sub) & 0xFFu) << 16) | (br[j] >> 16 << 24);
                }
            }
            __syncthreads();
            // Position by position: the lanes of a warp rank neighbours, and
            // what they write lands within a bin of where they are.
            uint32_t* out = d.payload_out + pos;
#pragma unroll 2
            for (uint32_t p = t; p < len; p += LOC_BLOCK) {
                const uint32_t meta = smeta[p], c = (meta >> 16) & 0xFFu, i = meta & 0xFFFFu;
                const uint32_t q0 = p - (meta >> 24);
                uint32_t at = q0;
                if (c > 1) {
                    const K k = skey[p];
                    for (uint32_t q = q0; q < q0 + c; ++q) {
                        const K o = skey[q];
                        at += o < k;
                        if (o == k && q != p) at += (smeta[q] & 0xFFFFu) < i;
                    }
                }
                out[at] = spay[i];
            }
            pos += len;
            __syncthreads();
        }
    }
}

// Dynamic shared memory of the local step.
template <typename K>
constexpr size_t local_smem() {
    return (size_t)LOC_BLOCK * KeyTraits<K>::LOC_ITEMS * (sizeof(K) + 4 + 4) + LOC_WORDS * 6;
}

template <typename K>
bolt_status run_sort(bolt_ctx* ctx, cudaStream_t s, const SortSpec& sp) {
    constexpr int NP = KeyTraits<K>::NPASS;
    constexpr int SORT_TILE = KeyTraits<K>::TILE;
    const int nseg = (int)sp.segs.size();
    if (nseg == 0) return BOLT_OK;
    std::vector<SegDesc> segs(nseg);
    std::vector<uint32_t> begins(3 * (nseg + 1));
    uint64_t total_n = 0, items = 0, hitems = 0, litems = 0;
    // Rows of one local work item: a few chunks, so that finding its ends is
    // a small part of it, but enough items for every CTA.
    uint64_t sum_n = 0;
    for (const SortSegment& g : sp.segs) sum_n += g.n;
    const uint64_t loc_range = std::min<uint64_t>(std::max<uint64_t>(sum_n / ((uint64_t)ctx->num_sms * 8) & ~1023ull, 4096), 32768);
    for (int i = 0; i < nseg; ++i) {
        const SortSegment& g = sp.segs[i];
        if (g.n >= (1ull << 30))
            return fail(ctx, BOLT_DECLINE, "radix sort: %llu rows exceed the 2^30 row limit", (ull)g.n);
        if (!g.payload_out && g.n) return fail(ctx, BOLT_ERR_INVALID, "radix sort: no payload output");
        segs[i] = SegDesc{g.keys, g.payload_in, g.payload_out, g.n_dev, g.n, total_n, (uint32_t)items, (uint32_t)hitems,
                          (uint32_t)litems};
        begins[i] = (uint32_t)items;
        begins[nseg + 1 + i] = (uint32_t)hitems;
        begins[2 * (nseg + 1) + i] = (uint32_t)litems;
        total_n += g.n;
        items += (g.n + SORT_TILE - 1) / SORT_TILE;
        hitems += (g.n + HIST_CHUNK - 1) / HIST_CHUNK;
        litems += (g.n + loc_range - 1) / loc_range;
    }
    begins[nseg] = (uint32_t)items;
    begins[2 * nseg + 1] = (uint32_t)hitems;
    begins[3 * nseg + 2] = (uint32_t)litems;
    if (items >= (1ull << 31)) return fail(ctx, BOLT_DECLINE, "radix sort: too many tiles");
    if (items == 0) return BOLT_OK;

    SortArgs a{};
    a.src = sp.src;
    a.desc = sp.descending;
    a.indirect = sp.indirect;
    a.nseg = nseg;
    a.total_items = (uint32_t)items;
    a.total_hist_items = (uint32_t)hitems;
    a.total_loc_items = (uint32_t)litems;
    a.loc_range = (uint32_t)loc_range;
    a.lb_stride = items * 256;
    const uint64_t nb = total_n ? total_n : 1;
    const bool many = nseg > 1;
    SegDesc* d_segs = many ? (SegDesc*)arena_alloc(ctx, sizeof(SegDesc) * nseg) : nullptr;
    uint32_t* d_begins = many ? (uint32_t*)arena_alloc(ctx, 4 * begins.size()) : nullptr;
    a.kA = arena_alloc(ctx, nb * sizeof(K));
    a.kB = arena_alloc(ctx, nb * sizeof(K));
    a.pA = (uint32_t*)arena_alloc(ctx, nb * 4);
    a.pB = (uint32_t*)arena_alloc(ctx, nb * 4);
    a.hist = (uint32_t*)arena_alloc(ctx, (uint64_t)nseg * NP * 256 * 4);
    a.digit_base = (uint32_t*)arena_alloc(ctx, (uint64_t)nseg * NP * 256 * 4);
    a.plan = (SegPlan*)arena_alloc(ctx, (uint64_t)nseg * sizeof(SegPlan));
    a.lookback = (uint32_t*)arena_alloc(ctx, 2 * a.lb_stride * 4);
    a.tile_ctr = (uint32_t*)arena_alloc(ctx, 64);
    constexpr uint64_t LOC_CAP = (uint64_t)LOC_BLOCK * KeyTraits<K>::LOC_ITEMS;
    a.max_longs = (uint32_t)(sum_n / LOC_CAP + 1);
    a.longs = reinterpret_cast<LongRun*>(a.lookback);
    static_assert(sizeof(LongRun) * 2 <= 256 * 4 && LOC_CAP >= (uint64_t)SORT_TILE, "the look-back words of a sort hold its long runs");
    a.status = ctx->d_status;
    if ((many && (!d_segs || !d_begins)) || !a.kA || !a.kB || !a.pA || !a.pB || !a.hist || !a.digit_base || !a.plan ||
        !a.lookback || !a.tile_ctr)
        return fail(ctx, BOLT_ERR_CAPACITY, "radix sort: scratch arena too small for %llu rows", (ull)total_n);
    a.segs = d_segs;
    a.seg0 = segs[0];
    if (many) {
        a.item_begins = d_begins;
        a.hist_begins = d_begins + nseg + 1;
        a.loc_begins = d_begins + 2 * (nseg + 1);
        bolt_status st = stage_upload(ctx, s, d_segs, segs.data(), sizeof(SegDesc) * nseg);
        if (st != BOLT_OK) return st;
        st = stage_upload(ctx, s, d_begins, begins.data(), 4 * begins.size());
        if (st != BOLT_OK) return st;
    }
    BOLT_CUDA(ctx, cudaMemsetAsync(a.hist, 0, (uint64_t)nseg * NP * 256 * 4, s));
    const unsigned hb = (unsigned)std::min<uint64_t>(hitems, (uint64_t)ctx->num_sms * 8);
    sort_hist_kernel<K><<<hb, HIST_BLOCK, 0, s>>>(a);
    BOLT_CUDA(ctx, smem_optin(sort_plan_kernel<K>, ctx));
    sort_plan_kernel<K><<<nseg, PLAN_BLOCK, 2 * PLAN_SAMPLES * 12, s>>>(a);
    ctx->last_launches += 2;
    const size_t dyn = (sizeof(K) + 5) * SORT_TILE;
    BOLT_CUDA(ctx, smem_optin(sort_pass_kernel<K>, ctx));
    const unsigned pg = (unsigned)std::min<uint64_t>(items, (uint64_t)ctx->num_sms * 3);
    for (int p = 0; p < NP; ++p) {
        sort_pass_kernel<K><<<pg, SORT_BLOCK, dyn, s>>>(a, p);
        ctx->last_launches++;
    }
    BOLT_CUDA(ctx, smem_optin(sort_local_kernel<K>, ctx));
    const unsigned lg = (unsigned)std::min<uint64_t>(litems, (uint64_t)ctx->num_sms * 2);
    sort_local_kernel<K><<<lg, LOC_BLOCK, local_smem<K>(), s>>>(a);
    ctx->last_launches++;
    if (sum_n > LOC_CAP) {
        BOLT_CUDA(ctx, smem_optin(sort_long_kernel<K>, ctx));
        const unsigned rg = (unsigned)std::min<uint64_t>(sum_n / LOC_CAP, (uint64_t)ctx->num_sms);
        sort_long_kernel<K><<<rg, LOC_BLOCK, local_smem<K>(), s>>>(a);
        ctx->last_launches++;
    }
    BOLT_CUDA(ctx, cudaGetLastError());
    return BOLT_OK;
}

}  // namespace

uint64_t radix_sort_scratch(uint64_t total_n, uint64_t nseg, int32_t src) {
    const uint64_t ksz = (src == SRC_I32 || src == SRC_F32 || src == SRC_U32) ? 4 : 8;
    const uint64_t items = total_n / SORT_TILE_MIN + nseg + 1;
    return 2 * total_n * (ksz + 4) + 2 * items * 256 * 4 + nseg * (2 * 8 * 256 * 4 + 96) + 64 * 1024;
}

bolt_status radix_sort(bolt_ctx* ctx, cudaStream_t s, const SortSpec& sp) {
    switch (sp.src) {
    case SRC_I32:
    case SRC_F32:
    case SRC_U32:
        return run_sort<uint32_t>(ctx, s, sp);
    case SRC_I64:
    case SRC_F64:
    case SRC_U64_KEYS:
        return run_sort<ull>(ctx, s, sp);
    }
    return fail(ctx, BOLT_ERR_INVALID, "radix sort: unknown key source %d", sp.src);
}

}  // namespace bolt

// ---------------------------------------------------------------------------
// ORDER BY entry points
// ---------------------------------------------------------------------------
#include "compact.cuh"

using namespace bolt;

namespace {

int sort_src_of(int dt) {
    switch (dt) {
    case BOLT_I32: return SRC_I32;
    case BOLT_I64: return SRC_I64;
    case BOLT_F32: return SRC_F32;
    case BOLT_F64: return SRC_F64;
    case BOLT_U32: return SRC_U32;
    }
    return -1;
}

}  // namespace

extern "C" bolt_status bolt_radix_sort_perm_multi(bolt_ctx* ctx, const bolt_col_view* keys, int32_t n_keys,
                                                  const int32_t* descending, const int32_t* nulls_first,
                                                  bolt_col_mut* perm, uint32_t flags, bolt_stream stream) {
    if (!ctx) return BOLT_ERR_INVALID;
    if (!keys || n_keys < 1 || !perm || !descending || !nulls_first)
        return fail(ctx, BOLT_ERR_INVALID, "ORDER BY: bad arguments");
    cudaStream_t s = (cudaStream_t)stream;
    const uint64_t n = keys[0].len;
    for (int k = 0; k < n_keys; ++k) {
        if (keys[k].len != n) return fail(ctx, BOLT_ERR_INVALID, "ORDER BY: key lengths differ");
        if (sort_src_of(keys[k].dtype) < 0) return fail(ctx, BOLT_DECLINE, "ORDER BY: key dtype %d", keys[k].dtype);
        if (!col_aligned(keys[k].data, keys[k].dtype))
            return fail(ctx, BOLT_ERR_INVALID, "ORDER BY: key %d is not aligned to its element width", k);
    }
    if (perm->dtype != BOLT_U32 || perm->cap < n) return fail(ctx, BOLT_ERR_CAPACITY, "ORDER BY: permutation output too small");
    if (n >= (1ull << 30)) return fail(ctx, BOLT_DECLINE, "ORDER BY: %llu rows exceed 2^30", (ull)n);
    bolt_status st = call_begin(ctx, flags, s);
    if (st != BOLT_OK) return st;
    uint32_t* out = (uint32_t*)perm->data;
    // Ping-pong between the caller's output and one scratch array so the
    // last (most significant) key writes the caller's buffer.
    uint32_t* tmp = n_keys > 1 ? (uint32_t*)arena_alloc(ctx, (n ? n : 1) * 4) : nullptr;
    ull* cnt = (ull*)arena_alloc(ctx, 256);
    if ((n_keys > 1 && !tmp) || !cnt) return fail(ctx, BOLT_ERR_CAPACITY, "ORDER BY: scratch arena too small");
    const uint32_t* cur = nullptr;  // nullptr = identity order
    kernel_mark_begin(ctx, flags, s);
    for (int k = n_keys - 1; k >= 0; --k) {
        uint32_t* dst = ((n_keys - 1 - k) % 2 == (n_keys - 1) % 2) ? out : tmp;
        const uint64_t mark = ctx->arena_used;
        const bolt_col_view& key = keys[k];
        SortSpec sp;
        sp.src = sort_src_of(key.dtype);
        sp.descending = descending[k];
        SortSegment seg;
        seg.keys = key.data;
        if (!key.validity) {
            seg.payload_in = cur;
            sp.indirect = cur != nullptr;
            seg.n = n;
            seg.payload_out = dst;
            sp.segs.push_back(seg);
            st = radix_sort(ctx, s, sp);
            if (st != BOLT_OK) return st;
        } else {
            // Stable NULL partition: valid rows are sorted, NULL rows keep
            // their current relative order and go first or last.
            uint32_t* valid_ids = (uint32_t*)arena_alloc(ctx, (n ? n : 1) * 4);
            if (!valid_ids) return fail(ctx, BOLT_ERR_CAPACITY, "ORDER BY: scratch arena too small");
            st = null_split_enqueue(ctx, s, n, key.validity, cur, valid_ids, dst, nulls_first[k] != 0, cnt);
            if (st != BOLT_OK) return st;
            BOLT_CUDA(ctx, cudaMemcpyAsync(ctx->h_words, cnt, 8, cudaMemcpyDeviceToHost, s));
            BOLT_CUDA(ctx, cudaStreamSynchronize(s));
            const ull nv = ctx->h_words[0];
            const uint64_t nn = n - nv;
            seg.payload_in = valid_ids;
            sp.indirect = 1;
            seg.n = nv;
            seg.payload_out = dst + (nulls_first[k] ? nn : 0);
            sp.segs.push_back(seg);
            st = radix_sort(ctx, s, sp);
            if (st != BOLT_OK) return st;
        }
        ctx->arena_used = mark;
        cur = dst;
    }
    kernel_mark_end(ctx, flags, s);
    if (flags & BOLT_FLAG_ASYNC) return call_end(ctx, flags, s);
    uint32_t f = 0;
    st = call_finish(ctx, flags, s, nullptr, 0, &f);
    if (st != BOLT_OK) return st;
    return flags_to_status(ctx, f, "ORDER BY");
}

extern "C" bolt_status bolt_radix_sort_perm(bolt_ctx* ctx, const bolt_col_view* key, int32_t descending,
                                            int32_t nulls_first, bolt_col_mut* perm, uint32_t flags,
                                            bolt_stream stream) {
    return bolt_radix_sort_perm_multi(ctx, key, 1, &descending, &nulls_first, perm, flags, stream);
}
