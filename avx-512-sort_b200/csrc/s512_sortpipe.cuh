// s512_sortpipe.cuh -- partition-then-sort pipeline for one GPU.
//
// The reference sorts by recursive two-way partitioning (Partition512,
// sort512.hpp:5729-5912, driven by CoreSort 5947-5958 with the pseudo-median
// pivot of CoreSortGetPivot 5916-5927) down to leaves of at most 16 vectors
// (SortLimite = 16*64/sizeof(T), 5949), which SmallSort16V sorts with bitonic
// networks.  This file keeps that method and widens each step for a GPU:
//
//   * a pivot becomes up to 255 splitters drawn from a random sample of the
//     segment, so one partition pass splits a segment into up to 256 buckets
//     instead of 2; they lie between value slots where the sample is spread
//     finely enough over those, else on keys of the sorted sample;
//   * splitter values that repeat in the sample get an equality bucket (keys
//     equal to that value need no further sorting), which removes the
//     reference's quadratic behaviour on few-distinct and sorted inputs;
//   * the partition pass is out of place and "one sweep": every tile of keys
//     gathers its keys by bucket in shared memory, reserves its share of each
//     bucket's output region with one atomic add per bucket, then writes each
//     bucket's keys there.  Bucket b of a
//     segment is written into a region whose capacity comes from the sample
//     (a 6-sigma bound); a bucket that outgrows it is reported and the level
//     is redone with exact counts;
//   * buckets at most a leaf's capacity are sorted in shared memory (one warp
//     and the bitonic networks of s512_bitonic.cuh up to 256 keys, one block
//     and the slot sort of s512_slotsort.cuh above, by size class) and written
//     to their final place; larger buckets become the segments of the next
//     partition level.
#pragma once

#include <cstddef>
#include <type_traits>

#include "s512_slotsort.cuh"

namespace s512 {

constexpr int NB = 256;            // buckets per segment per pass (max)
constexpr int SAMPLE_N = 16384;    // keys sampled per segment
constexpr int COPY_CHUNK = 16384;  // equality buckets are copied in chunks of this size
constexpr int SPLIT_SLOTS = 4096;  // value slots of the splitter lookup table
constexpr int DIRECT_SLOTS = 16384;  // value slots of the direct table (segments split at slot boundaries)

// A segment to partition at some level.
struct SegDesc {
    uint64_t in_off;     // first key in the level's input buffer
    uint64_t count;      // number of keys
    uint64_t final_off;  // where the segment's keys end in the final output
    uint64_t out_base;   // start of the segment's bucket regions in the level's output
    uint32_t tile_start; // first global tile index of the segment
    uint32_t ntiles;
};

// What finds the bucket of a segment's keys.
enum : uint32_t { ROUTE_SPLIT = 0, ROUTE_LEARNED = 1, ROUTE_TABLE = 2, ROUTE_LINEAR = 3 };

// Slot of a key in the direct table: its offset from lo, cut to 32 bits, times
// a fixed-point factor.  fast() is right for keys in [lo, lo + range] and sets
// `out` for any below lo or too far above; slot() is right for all (keys
// outside clamp to the ends).  Both stay below DIRECT_SLOTS for any key.
template <typename K>
struct DirectMap {
    K lo;
    uint32_t sh, mul;
    uint32_t dmax;   // cut offset of the upper bound
    uint32_t hmax;   // 64-bit keys: its high word
    __device__ __forceinline__ uint32_t cut(K d) const {
        if constexpr (sizeof(K) == 8)
            return min(__funnelshift_rc((uint32_t)d, (uint32_t)((uint64_t)d >> 32), sh), dmax);  // sh <= 32
        else
            return min((uint32_t)d, dmax);
    }
    __device__ __forceinline__ bool outside(K d) const {
        if constexpr (sizeof(K) == 8) return (uint32_t)((uint64_t)d >> 32) > hmax;
        else return (uint32_t)d > dmax;
    }
    __device__ __forceinline__ uint32_t fast(K x, bool& out) const {
        const K d = x - lo;
        out |= outside(d);
        return __umulhi(cut(d), mul);
    }
    __device__ __forceinline__ uint32_t slot(K x) const {
        const K d = x < lo ? K(0) : x - lo;
        return __umulhi(outside(d) ? dmax : cut(d), mul);
    }
    // the smallest key of slot s or above (s at most slot(lo + range), not 0)
    __device__ __forceinline__ K first_key(uint32_t s) const {
        const uint32_t d = (uint32_t)((((uint64_t)s << 32) + mul - 1) / mul);
        return lo + ((K)d << sh);
    }
};

// Splitters of one segment and the layout of its bucket regions.
template <typename K>
struct SplitSet {
    K tree[NB];            // Eytzinger tree of the unique splitters, nodes 1..255, padded with max
                           // (the exact-count fallback's search; the pass uses slot_tab)
    K uniq[NB];            // unique splitters in ascending order (padded with max)
    uint64_t region_off[NB];  // bucket region start, relative to SegDesc::out_base
    uint64_t region_cap[NB];  // bucket region capacity (keys)
    uint8_t range_b[NB];   // bucket of keys with lower_bound index j that are not equal to uniq[j]
    uint8_t eq_b[NB];      // bucket of keys equal to uniq[j] when splitter j has an equality bucket
    uint32_t eq_mask[NB / 32];     // splitter j has an equality bucket
    uint32_t bucket_eq[NB / 32];   // bucket b is an equality bucket
    uint32_t nbuckets;
    uint32_t has_eq;
    uint32_t nuniq;
    uint32_t pad_;
    // Lookup table over the sample's value range: keys are clamped to
    // [slot_map.lo, slot_hi] and mapped to SPLIT_SLOTS slots by slot_map.
    // Entry s packs lo | cnt << 8: lo = the number of unique splitters whose
    // slot is below s, cnt = how many share slot s.  A key of slot s has lo
    // splitters below it for sure and still has to be compared with
    // uniq[lo .. lo+cnt) -- none for most keys (255 splitters, 4096 slots).
    SlotMap<K> slot_map;
    K slot_hi;
    alignas(16) uint16_t slot_tab[SPLIT_SLOTS + 8];
    // A segment whose sample spreads over many slots is split at slot
    // boundaries (route): a key's bucket is then dir_tab[dir_map(key)], or
    // dir_map(key) itself where the sample is spread evenly, with no splitter
    // left to compare (uniq holds the same boundaries as keys).
    uint32_t route;      // ROUTE_*
    DirectMap<K> dir_map;
    alignas(16) uint8_t dir_tab[DIRECT_SLOTS];
};

// A bucket that a leaf kernel sorts (or copies) into its final place.
template <typename K>
struct LeafItem {
    const K* src;        // encoded keys in a level buffer
    uint64_t dst;        // index of the first key in the caller's output
    uint32_t count;
    uint32_t pad_;
};

// Leaf size classes.  Class 0 is one warp per bucket (a 256-key bitonic
// leaf); the others are one block per bucket (the slot sort of
// s512_slotsort.cuh, with the bitonic + merge-path block sort for uneven
// buckets).  A bucket's class is the smallest that holds it; the classes
// above 4096 are close together, because small blocks sort their keys faster
// (more buckets in flight per SM) and a bucket's keys should fill most of its
// class's slots.  The copy list holds equality buckets.
constexpr int NCLASS = 9;
constexpr int CLS_COPY = NCLASS;  // index of the copy list
__host__ __device__ constexpr int class_cap(int c) {
    return c == 0 ? 256 : c == 1 ? 1024 : c == 2 ? 2048 : c == 3 ? 4096 : c == 4 ? 4608 : c == 5 ? 5120
         : c == 6 ? 6144 : c == 7 ? 8192 : 16384;
}
__host__ __device__ constexpr uint32_t leaf_max(int /*key_bytes*/) { return 16384u; }
__host__ __device__ inline int class_of(int /*key_bytes*/, uint32_t count) {
    int c = 0;
    while (c < NCLASS - 1 && (uint32_t)class_cap(c) < count) ++c;
    return c;
}

// Number of buckets to aim for in a segment of `count` keys: enough that the
// average bucket is ~leaf_max/4, at most 256.
__host__ __device__ inline int target_buckets(int key_bytes, uint64_t count) {
    uint64_t want = (count * 4 + leaf_max(key_bytes) - 1) / leaf_max(key_bytes);
    if (want < 2) want = 2;
    if (want > NB) want = NB;
    return (int)want;
}

// Keys sampled from a segment that will be split into nb buckets: about 128
// per bucket (so a bucket's sample count is ~128 and its capacity bound ~1.6x
// its expected size), between 2048 and SAMPLE_N.
__host__ __device__ inline uint32_t sample_size(int nb) {
    uint32_t m = 128u * (uint32_t)nb;
    if (m < 2048u) m = 2048u;
    if (m > (uint32_t)SAMPLE_N) m = SAMPLE_N;
    return m;
}

// Upper bound of the total region capacity the splitter kernel may lay out
// for a segment of `count` keys (see splitter_kernel): 2.01*count + 4096.
__host__ __device__ inline uint64_t region_bound(uint64_t count) {
    return count * 2 + count / 100 + 4096;
}

// Level control block (device); read back by the host after each level.
struct LevelCtl {
    uint32_t tile_counter;
    uint32_t err;
    uint32_t n_next;          // segments for the next level
    uint32_t n_items[NCLASS + 1];
    uint32_t ntiles_next;
    uint64_t next_keys;       // keys in next-level segments
    uint64_t bound_next;      // region bound of the next level
    uint32_t max_bucket;      // largest bucket seen this level
    uint32_t nonempty;        // non-empty buckets this level
    uint64_t level_keys;      // keys partitioned this level
    uint32_t learned_used;    // segments routed by their learned model
    uint32_t plain_used;      // segments routed by the splitter tree
    uint32_t learned_fitted;  // segments whose learned model was trained
    uint32_t model_imb_bits;  // largest sample imbalance of a trained model (float bits)
    uint32_t n_uneven[NCLASS];  // leaves handed from the slot sort to the block sort
    uint32_t never_set;       // testing: a flag nothing writes (the injected wait)
    uint32_t blocks_done;     // leaf_any_kernel: blocks that have ended
    double bucket_sq;         // sum of squared non-empty bucket sizes this level
};

// ===========================================================================
// 1. Sampling: per segment, up to SAMPLE_N keys at hashed positions (with
// replacement), sorted, and the splitters and bucket regions they give

template <typename F>
__device__ __forceinline__ uint32_t first_index(uint32_t n, F past) {  // first i in [0, n) with past(i), else n
    uint32_t lo = 0, hi = n;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (past(mid)) hi = mid; else lo = mid + 1;
    }
    return lo;
}

// Scratch of make_splitters.
template <typename K>
struct SplitScratch {
    K cand[NB], uniq[NB];
    uint64_t cap[NB];
    uint64_t wtot64[NB / 32];
    uint32_t eqf[NB], sk[NB];
    uint32_t wtot[NB / 32];
    uint32_t beq[NB / 32];
    uint32_t total_u, total_eq;
};

// Region capacity of a bucket that holds cnt of the m samples of a segment of
// `count` keys (scale = count / m): 6 sigma above its expected size.
__device__ __forceinline__ uint64_t bucket_cap(uint32_t cnt, double scale, uint64_t count) {
    const float v = (float)cnt + 6.0f * sqrtf((float)cnt + 1.0f) + 16.0f;
    uint64_t cap = (uint64_t)((double)v * scale) + 1;
    if (cap > count) cap = count;
    return (cap + 15) & ~15ull;
}

// Region offsets, the splitters and their search tree, and the equality masks
// from w.cap, w.uniq and w.beq (complete: a barrier behind them).
template <typename K>
__device__ void write_layout(SplitSet<K>* out, SplitScratch<K>& w, bool my_eq) {
    const int t = threadIdx.x;
    const uint64_t my_cap = t < NB ? w.cap[t] : 0ull;
    const uint64_t off = block_exclusive_scan_first<NB, uint64_t>(my_cap, w.wtot64, (uint64_t*)nullptr);
    if (t < NB) {
        out->region_off[t] = off;
        out->region_cap[t] = my_cap;
        // Eytzinger tree over uniq[0..254]: node i at depth d has in-order index
        // (2*(i - 2^d) + 1) * 2^(7-d) - 1.
        if (t >= 1) {
            const int d = 31 - __clz(t);
            const int io = (2 * (t - (1 << d)) + 1) * (1 << (7 - d)) - 1;
            out->tree[t] = w.uniq[io];
        } else {
            out->tree[0] = KeyMax<K>::value;
        }
        out->uniq[t] = w.uniq[t];
        const unsigned bal_eq = __ballot_sync(0xFFFFFFFFu, my_eq);
        if ((t & 31) == 0) out->eq_mask[t >> 5] = bal_eq;
        if (t < NB / 32) out->bucket_eq[t] = w.beq[t];
    }
}

// Splitters and bucket regions of a segment of `count` keys from its m sorted
// samples smp(0..m).  Every thread of the block calls it (a multiple of 32
// threads, at least NB).
template <typename K, typename Smp>
__device__ void make_splitters(Smp smp, uint32_t m, uint64_t count, int nb, SplitSet<K>* out, SplitScratch<K>& w) {
    const int t = threadIdx.x;
    const int ncand = nb - 1;

    // candidate splitters at the sample quantiles
    K c = KeyMax<K>::value;
    if (t < ncand) c = smp((uint32_t)(((uint64_t)(t + 1) * m) / nb) - 1);
    if (t < NB) w.cand[t] = c;
    __syncthreads();
    const bool valid = t < ncand;
    const bool first = valid && (t == 0 || w.cand[t] != w.cand[t - 1]);
    const bool dup = valid && ((t > 0 && w.cand[t] == w.cand[t - 1]) || (t + 1 < ncand && w.cand[t] == w.cand[t + 1]));
    const uint32_t j = block_exclusive_scan_first<NB, uint32_t>(first ? 1u : 0u, w.wtot, &w.total_u);
    if (first) {
        w.uniq[j] = c;
        w.eqf[j] = dup ? 1u : 0u;
    }
    __syncthreads();
    const uint32_t K_u = w.total_u;
    if (t >= (int)K_u && t < NB) {
        w.uniq[t] = KeyMax<K>::value;
        w.eqf[t] = 0;
    }
    __syncthreads();
    // splitter lookup table over [sample min, sample max]
    const SlotMap<K> f = make_slot_map<K>(smp(0), smp(m - 1) - smp(0), (uint32_t)SPLIT_SLOTS);
    if (t < NB) w.sk[t] = t < (int)K_u ? f(w.uniq[t]) : 0xFFFFFFFFu;
    if (t == 0) {
        out->slot_map = f;
        out->slot_hi = smp(m - 1);
    }
    __syncthreads();
    for (uint32_t s = t; s < (uint32_t)SPLIT_SLOTS + 8; s += blockDim.x) {
        // splitters with slot < s, and those of slot s
        const uint32_t lo = first_index(K_u, [&](uint32_t i) { return w.sk[i] >= s; });
        uint32_t cnt = 0;
        while (s < (uint32_t)SPLIT_SLOTS && lo + cnt < K_u && w.sk[lo + cnt] == s) ++cnt;
        out->slot_tab[s] = (uint16_t)(lo | (cnt << 8));
    }
    // bucket ids: range_j, then eq_j if splitter j has one; the last range bucket is K_u
    const uint32_t my_eq = (t < (int)K_u) ? w.eqf[t] : 0u;
    const uint32_t eq_before = block_exclusive_scan_first<NB, uint32_t>(my_eq, w.wtot, &w.total_eq);
    const uint32_t range_id = (uint32_t)t + eq_before;  // valid for t <= K_u
    const uint32_t nbk = K_u + 1 + w.total_eq;

    // sample counts per bucket -> capacities
    // range bucket j (t <= K_u): keys in (uniq[j-1], uniq[j]] or (uniq[j-1], uniq[j]) if eq_j
    const double scale = (double)count / (double)m;
    if (t < NB) {
        w.cap[t] = 0;
        if (t < NB / 32) w.beq[t] = 0;
        out->range_b[t] = t <= (int)K_u ? (uint8_t)range_id : (uint8_t)0;
        out->eq_b[t] = (uint8_t)(my_eq ? range_id + 1 : 0);
    }
    __syncthreads();
    if (t <= (int)K_u && t < NB) {
        auto below = [&](K v) { return first_index(m, [&](uint32_t i) { return !(smp(i) < v); }); };
        auto upto = [&](K v) { return first_index(m, [&](uint32_t i) { return v < smp(i); }); };
        const uint32_t lo = t == 0 ? 0u : upto(w.uniq[t - 1]);
        const uint32_t end = t == (int)K_u ? m : upto(w.uniq[t]);
        const uint32_t hi = my_eq ? below(w.uniq[t]) : end;
        w.cap[range_id] = bucket_cap(hi > lo ? hi - lo : 0u, scale, count);
        if (my_eq) {
            w.cap[range_id + 1] = bucket_cap(end - hi, scale, count);
            atomicOr(&w.beq[(range_id + 1) >> 5], 1u << ((range_id + 1) & 31));
        }
    }
    __syncthreads();
    write_layout<K>(out, w, my_eq != 0);
    if (t == 0) {
        out->nbuckets = nbk;
        out->has_eq = w.total_eq ? 1u : 0u;
        out->nuniq = K_u;
        out->route = ROUTE_SPLIT;
    }
}

// The splitters of a sorted sample in global memory (one segment per block).
template <typename K>
__global__ void __launch_bounds__(NB) splitter_kernel(const K* __restrict__ samples, const SegDesc* __restrict__ segs,
                                                      uint32_t nsegs, SplitSet<K>* __restrict__ splits,
                                                      int key_bytes) {
    __shared__ SplitScratch<K> w;
    const uint32_t s = blockIdx.x;
    if (s >= nsegs) return;
    const K* smp = samples + (size_t)s * SAMPLE_N;
    const uint64_t count = segs[s].count;
    const int nb = target_buckets(key_bytes, count);
    make_splitters<K>([&](uint32_t i) { return smp[i]; }, sample_size(nb), count, nb, splits + s, w);
}

// Split a segment at slot boundaries, from the histogram of its samples over
// the slots: no sort, no splitter search, and the partition pass finds a key's
// bucket with one table byte, or none where the sample is spread evenly.  A
// slot goes to the bucket that the middle of its samples falls in (in rank),
// so bucket ids rise with the slots.  Returns
// false, with nothing written, when the sample is not spread finely enough
// over the slots: a slot that holds half a bucket's share (repeated values,
// clusters) would leave uneven buckets and needs splitters between keys.
// `smem` holds DIRECT_SLOTS counters, then the scratch.  Every thread calls it.
template <typename K, int THREADS, int IPT>
__device__ bool make_direct(const K (&key)[IPT], uint32_t m, uint64_t count, int nb, SplitSet<K>* out,
                            unsigned char* smem, SlotRed<K>& red) {
    constexpr int PER = DIRECT_SLOTS / THREADS;  // slots per thread
    static_assert(PER == 16, "a thread writes its slots' table bytes as one 16-byte word");
    struct Scratch {
        SplitScratch<K> w;
        uint32_t first_slot[NB + 1], rank0[NB + 1];  // per bucket: its first slot, the samples before it
        uint32_t sumsq;
        uint8_t last[THREADS];                       // per thread: the bucket of its last slot
        alignas(4) uint16_t before[DIRECT_SLOTS + 1];  // per slot: the samples before it
    };
    unsigned char* hist = smem;
    Scratch& d = *reinterpret_cast<Scratch*>(smem + DIRECT_SLOTS * sizeof(uint32_t));
    const unsigned t = threadIdx.x, lane = lane_id(), warp = t >> 5;
    auto quad = [&](int j) {
        return reinterpret_cast<uint4*>(hist + ctr_swizzle<PER>(t * PER * 4 + (uint32_t)j * 16));
    };
#pragma unroll
    for (int j = 0; j < PER / 4; ++j) *quad(j) = make_uint4(0u, 0u, 0u, 0u);
    K lo, range;
    block_bounds<K, THREADS, IPT>(key, m, red, lo, range);
    const SlotMap<K> f = make_slot_map<K>(lo, range, (uint32_t)DIRECT_SLOTS);
    if (f.direct) return false;  // fewer values than slots
    DirectMap<K> dm;
    dm.lo = lo;
    dm.sh = f.sh;
    dm.mul = f.mul;
    dm.dmax = (uint32_t)(range >> f.sh);
    dm.hmax = sizeof(K) == 8 ? (uint32_t)((uint64_t)range >> 32) : 0u;
    const uint32_t most = m / (uint32_t)nb / 2;  // samples allowed in a slot
    bool heavy = false;
#pragma unroll
    for (int r = 0; r < IPT; ++r) {
        if ((uint32_t)r * THREADS + t < m) {
            bool unused = false;
            const uint32_t a = ctr_swizzle<PER>(dm.fast(key[r], unused) * 4u);
            heavy |= atomicAdd(reinterpret_cast<uint32_t*>(hist + a), 1u) >= most;
        }
    }
    if (__syncthreads_or(heavy)) return false;

    // samples before each slot, and from them its bucket
    uint32_t sum = 0;
#pragma unroll
    for (int j = 0; j < PER / 4; ++j) {
        const uint4 q = *quad(j);
        sum += q.x + q.y + q.z + q.w;
    }
    uint32_t inc = sum;
#pragma unroll
    for (int k = 1; k < 32; k <<= 1) {
        const uint32_t o = __shfl_up_sync(0xFFFFFFFFu, inc, k);
        if (lane >= (unsigned)k) inc += o;
    }
    if (lane == 31) red.wtot[warp] = inc;
    if (t <= NB) {  // buckets that no slot starts are empty
        d.first_slot[t] = DIRECT_SLOTS;
        d.rank0[t] = m;
    }
    if (t < NB / 32) d.w.beq[t] = 0;
    __syncthreads();
    uint32_t run = __reduce_add_sync(0xFFFFFFFFu, lane < warp ? red.wtot[lane] : 0u) + inc - sum;
    const float per_rank = (float)nb / (float)(2 * m);
    // (counts below 2^15 and their products are exact enough in float that a
    // larger rank never gives a smaller bucket: the product is monotone)
    auto bucket = [&](uint32_t before, uint32_t c) {
        return min((uint32_t)((float)(2 * before + c) * per_rank), (uint32_t)(nb - 1));
    };
    uint32_t rank[PER], bk[PER];
#pragma unroll
    for (int j = 0; j < PER / 4; ++j) {
        const uint4 q = *quad(j);
        const uint32_t c[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            rank[4 * j + k] = run;
            bk[4 * j + k] = bucket(run, c[k]);
            run += c[k];
        }
    }
#pragma unroll
    for (int j = 0; j < PER / 2; ++j)
        reinterpret_cast<uint32_t*>(d.before)[t * (PER / 2) + j] = rank[2 * j] | (rank[2 * j + 1] << 16);
    if (t == 0) {
        d.before[DIRECT_SLOTS] = (uint16_t)m;
        d.sumsq = 0;
    }
    d.last[t] = (uint8_t)bk[PER - 1];
    __syncthreads();
    // Evenly spread?  Then nb equal slots need no table, and their sizes do
    // not carry the noise of the sample.  (Their sample counts are read off at
    // the nearest of the fine slots.)  Even: the counts' squared deviation is
    // about what chance gives (one share per bucket), and none stands out.
    auto fine = [&](uint32_t j) { return (j * (uint32_t)DIRECT_SLOTS + (uint32_t)nb - 1) / (uint32_t)nb; };
    uint32_t cl = 0;
    if (t < (unsigned)nb) cl = (uint32_t)d.before[fine(t + 1)] - (uint32_t)d.before[fine(t)];
    if (t < NB) {
        const uint32_t sq = __reduce_add_sync(0xFFFFFFFFu, cl * cl);
        if (lane == 0) atomicAdd(&d.sumsq, sq);
    }
    const float share = (float)m / (float)nb;
    const bool stands_out = __syncthreads_or((float)cl > 1.6f * share);
    const bool linear = !stands_out && (float)d.sumsq / share - (float)m <= 1.4f * (float)nb + 6.0f;
    if (linear) {
        dm.mul = make_slot_map<K>(lo, range, (uint32_t)nb).mul;
    } else {
        uint32_t pack[PER / 4];
#pragma unroll
        for (int j = 0; j < PER / 4; ++j)
            pack[j] = bk[4 * j] | (bk[4 * j + 1] << 8) | (bk[4 * j + 2] << 16) | (bk[4 * j + 3] << 24);
        reinterpret_cast<uint4*>(out->dir_tab)[t] = make_uint4(pack[0], pack[1], pack[2], pack[3]);
        uint32_t prev = t ? d.last[t - 1] : 0u;
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            for (; prev < bk[k]; ++prev) {
                d.first_slot[prev + 1] = t * PER + k;
                d.rank0[prev + 1] = rank[k];
            }
        }
        if (t == 0) d.rank0[0] = 0;
    }
    __syncthreads();
    if (t < NB) {
        const bool live = t < (unsigned)nb;
        const uint32_t c = linear ? cl : d.rank0[t + 1] - d.rank0[t];
        d.w.cap[t] = live ? bucket_cap(c, (double)count / (double)m, count) : 0ull;
        // splitter t: the last key before bucket t + 1 (slot 0 is always in
        // bucket 0: it holds less than half a bucket's samples)
        const uint32_t s = t + 1 >= (unsigned)nb ? 0xFFFFFFFFu : linear ? t + 1 : d.first_slot[t + 1];
        d.w.uniq[t] = s <= dm.slot(lo + range) ? dm.first_key(s) - 1 : KeyMax<K>::value;
        out->range_b[t] = live ? (uint8_t)t : (uint8_t)0;
        out->eq_b[t] = 0;
    }
    __syncthreads();
    write_layout<K>(out, d.w, false);
    if (t == 0) {
        out->nbuckets = (uint32_t)nb;
        out->has_eq = 0;
        out->nuniq = (uint32_t)nb - 1;
        out->route = linear ? ROUTE_LINEAR : ROUTE_TABLE;
        out->dir_map = dm;
    }
    return true;
}

// Start of a level: keys sampled from every segment, `parts` blocks per
// segment (random reads are bound by how many one SM can have outstanding, so
// they are spread over the chip: 16384 reads by one block take 13 us to 33 us,
// by 64 blocks 2.2 us).  The level's control block and fill counters are zeroed
// on the way, and the segment of a level that is one `whole` array is written
// (as launches of their own these cost a small level 4 us).
template <typename Codec>
__global__ void __launch_bounds__(NB) sample_kernel(Codec in, SegDesc* __restrict__ segs, uint32_t parts,
                                                    typename Codec::Key* __restrict__ samples, uint64_t seed,
                                                    int key_bytes, LevelCtl* ctl, uint64_t* counts, int whole,
                                                    SegDesc first) {
    const uint32_t s = blockIdx.x / parts, part = blockIdx.x % parts;
    if (part == 0) counts[(size_t)s * NB + threadIdx.x] = 0;
    if (blockIdx.x == 0) {
        for (uint32_t i = threadIdx.x; i < sizeof(LevelCtl) / 4; i += NB) reinterpret_cast<uint32_t*>(ctl)[i] = 0;
        if (whole && threadIdx.x == 0) segs[0] = first;
    }
    const uint64_t in_off = whole ? first.in_off : segs[s].in_off, count = whole ? first.count : segs[s].count;
    const uint32_t m = sample_size(target_buckets(key_bytes, count));
#pragma unroll 4
    for (uint32_t i = part * NB + threadIdx.x; i < m; i += parts * NB)
        samples[(size_t)s * SAMPLE_N + i] =
            in.load(in_off + __umul64hi(mix64(seed ^ ((uint64_t)s << 32) ^ (uint64_t)i), count));
}

// Splitters and regions of every segment from its samples: one block of 1024
// threads per segment.  The work is a chain of latencies on one SM, so the
// sort of the sample is left out where its histogram will do (make_direct),
// and searches run in shared memory.  Sampling to splitters for one segment:
// int32 52 -> 11 us, 64-bit keys 58 -> 15 us; for the 256 segments of the
// second level of 2^28 doubles 165 -> 125 us (three kernels before, the
// sample sorted, written out and searched in L2).
constexpr int SAMPLE_THREADS = 1024;
constexpr int SAMPLE_IPT = SAMPLE_N / SAMPLE_THREADS;
template <typename K>
constexpr size_t split_smem() { return SlotSmem<K, SAMPLE_THREADS, SAMPLE_IPT>::bytes; }

template <typename K>
__global__ void __launch_bounds__(SAMPLE_THREADS)
    split_kernel(K* __restrict__ samples, const SegDesc* __restrict__ segs, SplitSet<K>* __restrict__ splits,
                 int key_bytes, int keep_sorted, int pairs) {
    using SM = SlotSmem<K, SAMPLE_THREADS, SAMPLE_IPT>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ SlotRed<K> red;
    const uint32_t s = blockIdx.x;
    const uint64_t count = segs[s].count;
    const int nb = target_buckets(key_bytes, count);
    const uint32_t m = sample_size(nb);
    K* g = samples + (size_t)s * SAMPLE_N;
    K key[SAMPLE_IPT];
#pragma unroll
    for (int r = 0; r < SAMPLE_IPT; ++r) {
        const uint32_t i = (uint32_t)r * SAMPLE_THREADS + threadIdx.x;
        if (i < m) key[r] = g[i];
    }
    if (make_direct<K, SAMPLE_THREADS, SAMPLE_IPT>(key, m, count, nb, splits + s, smem_raw, red)) return;
    __syncthreads();
    const K any = key[0];  // (m >= SAMPLE_THREADS)
    // sorted in registers and shared memory, where the splitters are searched;
    // back to global memory only for the learned fit
    const SlotPath how = block_slot_sort<K, SAMPLE_THREADS, SAMPLE_IPT, SLOT_REFINE>(
        key, m, [&](uint32_t i, K x) { if (keep_sorted) g[i] = x; }, [] {}, [] {}, smem_raw, red, !pairs);
    __syncthreads();
    const K* sorted = reinterpret_cast<const K*>(smem_raw);
    static_assert(SM::padded_bytes + sizeof(SplitScratch<K>) <= SM::bytes, "the space behind the keys is reused");
    SplitScratch<K>& w = *reinterpret_cast<SplitScratch<K>*>(smem_raw + SM::padded_bytes);
    make_splitters<K>(
        [&](uint32_t i) { return how == SLOT_EQUAL ? any : sorted[how == SLOT_EVEN ? i : pidx(i)]; }, m, count, nb,
        splits + s, w);
}

// Bucket of key x under a split set held in shared memory.
template <typename K>
__device__ __forceinline__ uint32_t find_bucket(const K* __restrict__ tree, K x, bool has_eq,
                                                const K* __restrict__ uniq, const uint8_t* __restrict__ range_b,
                                                const uint8_t* __restrict__ eq_b, const uint32_t* __restrict__ eq_mask) {
    uint32_t i = 1;
#pragma unroll
    for (int d = 0; d < 8; ++d) i = 2 * i + (tree[i] < x ? 1u : 0u);
    const uint32_t j = i - 256;  // number of unique splitters < x
    if (!has_eq) return j;
    if (j < 255 && ((eq_mask[j >> 5] >> (j & 31)) & 1u) && uniq[j] == x) return eq_b[j];
    return range_b[j];
}

// A split set's slot map held in registers for a run of lookups: keys are
// clamped to [lo, lo + range] (one compare: x - lo wraps above range when
// x < lo), cut to 32 bits by a funnel shift and scaled.  Same slots as
// SlotMap::operator() on the clamped key.
template <typename K>
struct SlotRegs {
    K lo, range;
    uint32_t sh, mul;
    bool direct;
    __device__ __forceinline__ SlotRegs(const SlotMap<K>& f, K hi)
        : lo(f.lo), range(hi - f.lo), sh(f.sh), mul(f.mul), direct(f.direct != 0) {}
    __device__ __forceinline__ uint32_t operator()(K x) const {
        K d = x - lo;
        if (d > range) d = x < lo ? K(0) : range;
        uint32_t d32;
        if constexpr (sizeof(K) == 8)
            d32 = __funnelshift_rc((uint32_t)d, (uint32_t)(d >> 32), sh);  // sh <= 32
        else
            d32 = (uint32_t)d >> sh;
        return direct ? d32 : __umulhi(d32, mul);
    }
};

// Bucket of key x given its slot entry (see SplitSet::slot_tab).
template <typename K>
__device__ __forceinline__ uint32_t bucket_from_slot(uint32_t e, K x, bool has_eq, const K* __restrict__ uniq,
                                                     const uint8_t* __restrict__ range_b,
                                                     const uint8_t* __restrict__ eq_b,
                                                     const uint32_t* __restrict__ eq_mask) {
    uint32_t lo = e & 0xFFu;
    const uint32_t cnt = e >> 8;
    if (cnt) {
        if (cnt == 1) {  // one splitter shares the key's slot
            lo += uniq[lo] < x ? 1u : 0u;
        } else {
            uint32_t hi = lo + cnt;
            while (lo < hi) {
                const uint32_t mid = (lo + hi) >> 1;
                if (uniq[mid] < x) lo = mid + 1; else hi = mid;
            }
        }
    }
    const uint32_t j = lo;  // number of unique splitters < x
    if (!has_eq) return j;
    if (j < 255 && ((eq_mask[j >> 5] >> (j & 31)) & 1u) && uniq[j] == x) return eq_b[j];
    return range_b[j];
}

}  // namespace s512

#include "s512_learned.cuh"

namespace s512 {

// ===========================================================================
// 4. The partition pass (persistent; tiles claimed in runs)
//
// Every tile of keys is classified, ranked within its bucket by shared-memory
// atomics, put in its bucket's bin in shared memory and written out from
// there, a group of lanes per bin.  Where a tile's keys of bucket b go inside
// the bucket's region is reserved with one global atomic add per (tile,
// bucket) on the segment's fill counter of b: the pass is not stable (a
// bucket's keys land in the order their tiles reserved, and the leaves sort
// them anyway), so no tile ever waits for another and tiles may be processed
// in any order.  The counters end as the bucket sizes.  A reservation past the
// region's capacity (the sample's 6-sigma bound) drops the tile's keys of that
// bucket and reports an overflow; the level is then redone with exact counts.
//
// What bounds it is the shared-memory pipe (wavefronts per key), then issue
// slots; HBM is third.  So a key costs one random shared access for its bucket
// (none on ROUTE_LINEAR), one atomic for its rank and one store into its bin:
// a bin holds a fixed number of keys, about 2.5 times a bucket's share of the
// tile, so its place needs no scan and no lookup, and the write-out reads a
// bin's pointer and count once per group of lanes instead of a bucket id and a
// pointer per key.  A tile with a fuller bucket (sorted or skewed input) is
// staged compactly in bucket order instead, with a scan of the counts and a
// bucket id per key.
//
// The next tile's keys are loaded into registers as soon as the current ones
// are in their bins, a run of 512 * 8 bytes per load instruction of the block;
// the loads complete while the tile is reserved and written.  Three block
// barriers per tile: bins free | bins filled | places known; a warp that has
// written its bins classifies its next keys before it waits.  Two blocks share
// an SM, so one block's barrier phases overlap the other's memory traffic.
// (Loads must stay raw bits until then: encoding them where they are loaded
// made every thread wait there.  Bulk copies into shared memory, which this
// pass used before, cost two more shared wavefronts per 32 keys.)
// Measured, one pass over 2^28 doubles, floor 0.66 ms: level 0 (ROUTE_TABLE)
// 1.25 -> 1.20 ms, level 1 (ROUTE_LINEAR) 1.38 -> 1.17 ms; 1.58 and 1.64 ms
// when every key was clamped, compared with the splitters of its slot and
// staged with a bucket id.  2^20 int32: 29 -> 7.5 us (shorter claim runs).
constexpr int SEG_SMEM = 256;  // segment tables up to this size are searched in shared memory
// Consecutive tiles a block claims at once, at most: one segment's tables are
// loaded once per group, so levels with many segments take longer runs; a
// single segment takes short ones (a finer split of the last tiles among
// blocks).  A launch of few tiles takes shorter runs still, so that every
// block has some: 733 tiles of one segment 73 -> 31 us, 171 of 2^20 int32 37 -> 7.5 us
// against runs of 4 with two claimed at once.
constexpr uint32_t CLAIM_GROUP_ONE_SEG = 4;
constexpr uint32_t CLAIM_GROUP_MANY_SEGS = 16;
// Keys past the regions of a level buffer where a bucket that overflowed its
// region writes its keys of the tile (at most a tile's worth; tiles race
// there harmlessly: the level is redone with exact counts).
constexpr uint64_t JUNK_KEYS = 8192;

template <typename K>
struct PartArgs {
    const SegDesc* segs;
    uint32_t nsegs;               // segment count (host-known)
    const uint32_t* tile_seg;     // global tile -> segment (nullptr: single segment 0)
    const SplitSet<K>* splits;
    K* out;                       // level output buffer
    uint64_t junk;                // offset in out of the JUNK_KEYS overflow area
    unsigned long long* fill;     // nsegs * NB fill counters (zeroed); end as the bucket sizes
    LevelCtl* ctl;
    uint32_t ntiles;              // end of the launch's tiles (used when ntiles_dev is null)
    const uint32_t* ntiles_dev;   // tile count written by prepare_level_kernel
    uint32_t tile_first;          // first tile of the launch (a level fed in chunks launches per chunk)
    uint32_t* tile_counter;       // the launch's claim counter (zeroed)
    const LearnedSet<K>* learned; // per segment learned model (nullptr: splitters only)
    int inject_timeout;           // testing: tile 1 waits, with a short bound, on a flag nothing sets
};

// The routing tables of a plain split set, as the partition pass keeps them.
template <typename K>
struct PlainTables {
    K uniq[NB];
    uint8_t range_b[NB];
    uint8_t eq_b[NB];
    uint32_t eq_mask[NB / 32];
    SlotMap<K> fmap;
    K fhi;
    alignas(16) uint16_t tab[SPLIT_SLOTS + 8];
};

// The routing table of a segment split at slot boundaries.
template <typename K>
struct DirectTables {
    DirectMap<K> map;
    alignas(16) uint8_t tab[DIRECT_SLOTS];
};

// Bytes of a LearnedSet that inference reads (its leading fields).
template <typename K>
constexpr size_t learned_model_bytes() { return offsetof(LearnedSet<K>, region_off); }

// Keys a bin holds: about 2.5 times the even share of a tile (16 keys of 64
// bits, 24 of 32 bits), so that on evenly split keys a fuller one is rare (a
// bucket at 1.4 times its share overflows one tile in thousands) and two
// blocks fit an SM.  Odd, so that equal places of different bins, which fill
// at the same time, lie on different banks.
__host__ __device__ constexpr int bin_cap(int tile) { return (tile * 5 / 2 / NB) | 1; }
// A segment's tiles use the bins where that makes an average bin half full at
// most, and where places in its regions (region_bound: 2.01 times its keys)
// fit 32 bits.
__host__ __device__ constexpr bool use_bins(int tile, uint32_t nbuckets, uint64_t seg_count) {
    return (uint32_t)tile * 2 <= nbuckets * (uint32_t)bin_cap(tile) && seg_count <= 2000000000ull;
}

template <typename K, int THREADS, int IPT>
struct PartSmem {
    static constexpr int TILE = THREADS * IPT;
    static constexpr int CAP = bin_cap(TILE);
    struct Compact {
        K stage[TILE];
        uint8_t bkt[TILE];
    };
    union {
        alignas(16) K bins[NB * CAP];
        Compact c;
    } u;
    struct alignas(8) Bin {
        uint32_t place, count;    // where the bin's key 0 goes in the segment's regions, and its keys
    };
    union {
        Bin bin[NB];
        uint64_t ptr[NB];         // compact tiles: where the bucket would put the tile's position 0
    } w;
    uint64_t region_off[NB];
    uint64_t region_cap[NB];
    alignas(16) uint32_t hist[NB];
    alignas(16) uint32_t loc[NB];
    uint32_t seg_tile_start[SEG_SMEM];
    struct Tile {
        uint64_t first;           // its first key in the input
        uint32_t count;           // its keys (0: no more tiles)
        uint32_t seg, index, pad_;
    } tile[2];
    uint64_t out_base;
    uint32_t has_eq, route, bins;
    // a segment routes by one of these
    union {
        PlainTables<K> P;
        DirectTables<K> D;
        alignas(16) unsigned char model[learned_model_bytes<K>()];
    } T;
};

template <typename K, typename InCodec, int THREADS, int IPT>
__global__ void __launch_bounds__(THREADS, 1024 / THREADS) partition_kernel(PartArgs<K> a, InCodec in) {
    extern __shared__ __align__(128) unsigned char smem_part[];
    using SM = PartSmem<K, THREADS, IPT>;
    SM& sm = *reinterpret_cast<SM*>(smem_part);
    constexpr int TILE = THREADS * IPT;
    constexpr uint32_t CAP = SM::CAP;
    static_assert(TILE < (1 << 21), "rank and bucket share a 32-bit word");
    static_assert(TILE <= (int)JUNK_KEYS, "an overflowed bucket's keys of a tile fit the overflow area");
    static_assert(sizeof(typename SM::Compact) <= sizeof(K) * NB * CAP, "the compact stage fits the bins' space");
    static_assert(THREADS >= NB, "a thread per bucket");
    const int tid = threadIdx.x;
    const uint32_t ntiles = a.ntiles_dev ? *a.ntiles_dev : a.ntiles;
    const bool small_tab = a.tile_seg && a.nsegs <= (uint32_t)SEG_SMEM;
    const bool claimer = tid == THREADS - 1;  // (the last warp: the first ones reserve and scan)

    if (tid < NB) sm.hist[tid] = 0;
    if (small_tab)
        for (uint32_t i = tid; i < a.nsegs; i += THREADS) sm.seg_tile_start[i] = a.segs[i].tile_start;
    __syncthreads();

    auto seg_of = [&](uint32_t t) -> uint32_t {
        if (!a.tile_seg) return 0u;
        if (!small_tab) return a.tile_seg[t];
        uint32_t lo = 0, hi = a.nsegs;  // last segment whose tile_start <= t
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (sm.seg_tile_start[mid] <= t) lo = mid; else hi = mid;
        }
        return lo;
    };
    // The claimer takes claim_group consecutive tiles at a time: the first
    // group by the block's index, the others from the counter.  A group is
    // claimed with the last tile of the one before (the atomic's latency
    // passes while that tile is processed).
    const uint32_t most = a.nsegs > 1 ? CLAIM_GROUP_MANY_SEGS : CLAIM_GROUP_ONE_SEG;
    const uint32_t claim_group = min(max((ntiles - min(a.tile_first, ntiles)) / (gridDim.x * 2), 1u), most);
    uint32_t grp_next = a.tile_first + blockIdx.x * claim_group, grp_end = grp_next + claim_group, grp_ahead = 0;
    uint32_t c_seg = 0xFFFFFFFFu, c_tile0 = 0;
    uint64_t c_off = 0, c_count = 0;
    auto next_tile = [&](typename SM::Tile* slot) {
        if (grp_next == grp_end) {
            grp_next = grp_ahead;
            grp_end = grp_next + claim_group;
        }
        const uint32_t t = grp_next++;
        if (grp_next == grp_end)
            grp_ahead = a.tile_first + gridDim.x * claim_group + atomicAdd(a.tile_counter, claim_group);
        slot->count = 0;
        if (t >= ntiles) return;
        const uint32_t seg = seg_of(t);
        if (seg != c_seg) {  // (tiles come in runs of one segment)
            c_seg = seg;
            c_off = a.segs[seg].in_off;
            c_count = a.segs[seg].count;
            c_tile0 = a.segs[seg].tile_start;
        }
        const uint64_t at = (uint64_t)(t - c_tile0) * TILE;
        slot->first = c_off + at;
        slot->count = c_count - at < (uint64_t)TILE ? (uint32_t)(c_count - at) : (uint32_t)TILE;
        slot->seg = seg;
        slot->index = t;
    };
    if (claimer) {
        next_tile(&sm.tile[0]);
        next_tile(&sm.tile[1]);
    }
    __syncthreads();

    K key[IPT];  // the tile's keys, striped (element r*THREADS + tid); as stored until they are classified
    auto load = [&](uint64_t first, uint32_t cnt) {
        if (cnt == (uint32_t)TILE) {
#pragma unroll
            for (int r = 0; r < IPT; ++r) key[r] = in.raw(first + (uint32_t)(r * THREADS + tid));
        } else {
#pragma unroll
            for (int r = 0; r < IPT; ++r)
                if ((uint32_t)(r * THREADS + tid) < cnt) key[r] = in.raw(first + (uint32_t)(r * THREADS + tid));
        }
    };
    uint32_t cnt = sm.tile[0].count, seg = sm.tile[0].seg, index = sm.tile[0].index;
    load(sm.tile[0].first, cnt);
    uint32_t cached_seg = 0xFFFFFFFFu;

    for (uint32_t turn = 1; cnt != 0; turn ^= 1) {  // turn: the slot of the next tile
        if (seg != cached_seg) {
            // the segment's tables, read once per run of its tiles (the
            // previous tile's write-out reads none of them)
            const uint32_t route = a.learned && a.learned[seg].ok ? ROUTE_LEARNED : a.splits[seg].route;
            const SplitSet<K>& ss = a.splits[seg];
            const uint64_t* off = route == ROUTE_LEARNED ? a.learned[seg].region_off : ss.region_off;
            const uint64_t* cap = route == ROUTE_LEARNED ? a.learned[seg].region_cap : ss.region_cap;
            if (tid < NB) {
                sm.region_off[tid] = off[tid];
                sm.region_cap[tid] = cap[tid];
            }
            if (route == ROUTE_TABLE) {
                const uint4* src = reinterpret_cast<const uint4*>(ss.dir_tab);
                uint4* dst = reinterpret_cast<uint4*>(sm.T.D.tab);
                for (int i = tid; i < DIRECT_SLOTS / 16; i += THREADS) dst[i] = src[i];
            } else if (route == ROUTE_LEARNED) {
                const uint32_t* src = reinterpret_cast<const uint32_t*>(&a.learned[seg]);
                uint32_t* dst = reinterpret_cast<uint32_t*>(sm.T.model);
                for (uint32_t i = tid; i < learned_model_bytes<K>() / 4; i += THREADS) dst[i] = src[i];
            } else if (route == ROUTE_SPLIT) {
                if (tid < NB) {
                    sm.T.P.uniq[tid] = ss.uniq[tid];
                    sm.T.P.range_b[tid] = ss.range_b[tid];
                    sm.T.P.eq_b[tid] = ss.eq_b[tid];
                }
                if (tid < NB / 32) sm.T.P.eq_mask[tid] = ss.eq_mask[tid];
                const uint4* src = reinterpret_cast<const uint4*>(ss.slot_tab);
                uint4* dst = reinterpret_cast<uint4*>(sm.T.P.tab);
                for (int i = tid; i < (SPLIT_SLOTS + 8) * 2 / 16; i += THREADS) dst[i] = src[i];
            }
            if (tid == 0) {
                sm.out_base = a.segs[seg].out_base;
                sm.route = route;
                sm.bins = use_bins(TILE, route == ROUTE_LEARNED ? a.learned[seg].nbuckets : ss.nbuckets,
                                   a.segs[seg].count);
                if (route == ROUTE_TABLE || route == ROUTE_LINEAR) {
                    sm.T.D.map = ss.dir_map;
                } else if (route == ROUTE_SPLIT) {
                    sm.has_eq = ss.has_eq;
                    sm.T.P.fmap = ss.slot_map;
                    sm.T.P.fhi = ss.slot_hi;
                }
            }
            cached_seg = seg;
            __syncthreads();
        }
        if (a.inject_timeout && index == 1) {
            // injected failure: a wait on a flag that nothing sets, with a
            // short bound; the block then gives up and writes nothing more
            uint32_t spins = 0;
            while (!*(volatile uint32_t*)&a.ctl->never_set && ++spins < 1024u) __nanosleep(100);
            raise_error(&a.ctl->err, DEV_ERR_TIMEOUT);
            break;
        }

        // A. buckets and ranks.  All IPT bucket lookups first: they are
        // independent chains, so the scheduler can overlap them.
        uint32_t br[IPT];  // 4 * bucket | rank << 11
        bool over = !sm.bins;  // some bucket has more keys of the tile than a bin holds
        auto classify = [&](auto full) {
            constexpr bool FULL = decltype(full)::value;
            const uint32_t route = sm.route;
#pragma unroll
            for (int r = 0; r < IPT; ++r) key[r] = InCodec::enc(key[r]);
            if (route >= ROUTE_TABLE) {
                const DirectMap<K> dm = sm.T.D.map;
                bool out = false;
                // (lanes past the end look up stale register contents, in
                // bounds, and then carry the out-of-range bucket NB)
#pragma unroll
                for (int r = 0; r < IPT; ++r) br[r] = dm.fast(key[r], out);
                if (out) {  // a key outside the sample's range (2 in 16384 or so)
#pragma unroll
                    for (int r = 0; r < IPT; ++r) br[r] = dm.slot(key[r]);
                }
                if (route == ROUTE_TABLE) {
#pragma unroll
                    for (int r = 0; r < IPT; ++r) br[r] = sm.T.D.tab[br[r]];
                }
#pragma unroll
                for (int r = 0; r < IPT; ++r) br[r] <<= 2;
            } else if (route == ROUTE_LEARNED) {
#pragma unroll
                for (int r = 0; r < IPT; ++r)  // (only the model prefix of the LearnedSet is in shared memory)
                    if (FULL || (uint32_t)(r * THREADS + tid) < cnt)
                        br[r] = learned_bucket<K>(*reinterpret_cast<const LearnedSet<K>*>(sm.T.model), key[r]) << 2;
            } else {
                const bool has_eq = sm.has_eq != 0;
                const SlotRegs<K> fm(sm.T.P.fmap, sm.T.P.fhi);
#pragma unroll
                for (int r = 0; r < IPT; ++r) br[r] = sm.T.P.tab[fm(key[r])];  // slot entries first
#pragma unroll
                for (int r = 0; r < IPT; ++r)
                    if (FULL || (uint32_t)(r * THREADS + tid) < cnt)
                        br[r] = bucket_from_slot<K>(br[r], key[r], has_eq, sm.T.P.uniq, sm.T.P.range_b, sm.T.P.eq_b,
                                                    sm.T.P.eq_mask) << 2;
            }
            if (!FULL) {
#pragma unroll
                for (int r = 0; r < IPT; ++r)
                    if ((uint32_t)(r * THREADS + tid) >= cnt) br[r] = 4u * NB;
            }
            auto hist = [&](uint32_t b4) { return reinterpret_cast<uint32_t*>(reinterpret_cast<char*>(sm.hist) + b4); };
            // A warp whose 32 keys share a bucket (sorted or constant runs)
            // ranks them with one atomic instead of 32 on one address.  Whether
            // to look for that is decided once per tile from the warp's first
            // 32 keys: on unsorted input the check would cost a shuffle and a
            // vote per key and never pay.
            if (__all_sync(0xFFFFFFFFu, br[0] == __shfl_sync(0xFFFFFFFFu, br[0], 0))) {
#pragma unroll
                for (int r = 0; r < IPT; ++r) {
                    const uint32_t b0 = __shfl_sync(0xFFFFFFFFu, br[r], 0);
                    uint32_t rank = 0;
                    if (__all_sync(0xFFFFFFFFu, br[r] == b0)) {
                        if (b0 < 4u * NB) {
                            uint32_t basev = 0;
                            if (lane_id() == 0) basev = atomicAdd(hist(b0), 32u);
                            rank = __shfl_sync(0xFFFFFFFFu, basev, 0) + lane_id();
                        }
                    } else if (br[r] < 4u * NB) {
                        rank = atomicAdd(hist(br[r]), 1u);
                    }
                    br[r] |= rank << 11;
                    over |= rank >= CAP;
                }
            } else {
#pragma unroll
                for (int r = 0; r < IPT; ++r)
                    if (FULL || br[r] < 4u * NB) {
                        br[r] |= atomicAdd(hist(br[r]), 1u) << 11;
                        over |= br[r] >= (CAP << 11);
                    }
            }
        };
        if (cnt == (uint32_t)TILE) classify(std::true_type{});
        else classify(std::false_type{});
        __syncthreads();  // (1) the bins are free: the previous tile is written

        // B. the keys into their buckets' bins
        if (sm.bins) {
#pragma unroll
            for (int r = 0; r < IPT; ++r) {
                const uint32_t b4 = br[r] & 0x7FFu, rank = br[r] >> 11;
                if (b4 < 4u * NB && rank < CAP) sm.u.bins[(b4 >> 2) * CAP + rank] = key[r];
            }
        }
        const bool compact = __syncthreads_or(over);  // (2) bins and counts are complete

        // C. reserve the tile's share of each bucket's region
        uint32_t h = 0;
        unsigned long long off = 0;
        if (tid < NB) {
            h = sm.hist[tid];
            if (h) off = atomicAdd(&a.fill[(size_t)seg * NB + tid], (unsigned long long)h);
        }
        const uint32_t tile_cnt = cnt;
        auto advance = [&]() {  // the next tile's keys (the current ones are staged)
            const typename SM::Tile& nx = sm.tile[turn];
            cnt = nx.count;
            seg = nx.seg;
            index = nx.index;
            load(nx.first, cnt);
        };
        // where the bucket's keys of the tile go (an overflowed bucket's to the
        // overflow area past the regions: the level is redone)
        auto overflows = [&]() {
            const bool ovf = off + h > sm.region_cap[tid];
            if (ovf && h) raise_error(&a.ctl->err, DEV_ERR_OVERFLOW);
            return ovf;
        };
        if (!compact) {
            if (tid < NB) sm.hist[tid] = 0;
            advance();
            if (claimer) next_tile(&sm.tile[turn ^ 1]);
            if (tid < NB) {
                // (places fit 32 bits; an overflowed bucket is not written)
                typename SM::Bin o;
                o.place = (uint32_t)(sm.region_off[tid] + off);
                o.count = overflows() ? 0u : h;
                sm.w.bin[tid] = o;
            }
            K* const seg_out = a.out + sm.out_base;
            __syncthreads();  // (3) places known
            // D. each group of lanes writes out its bins
            constexpr int GL = sizeof(K) == 8 ? 16 : 32, NG = THREADS / GL;
            const uint32_t g = (uint32_t)tid / GL, l = (uint32_t)tid % GL;
#pragma unroll 4
            for (uint32_t b = g; b < (uint32_t)NB; b += NG) {
                const typename SM::Bin o = sm.w.bin[b];
                const K* src = sm.u.bins + b * CAP;
                K* dst = seg_out + o.place;
                if (l < o.count) dst[l] = src[l];
                if (l + GL < o.count) dst[l + GL] = src[l + GL];
                if (2 * GL < CAP && l + 2 * GL < o.count) dst[l + 2 * GL] = src[l + 2 * GL];
            }
            static_assert(CAP <= 3 * GL, "a bin is at most three keys per lane");
        } else {
            // the tile in bucket order: exclusive scan of the counts by warp 0
            if (tid < 32) {
                uint32_t v[NB / 32];
                uint32_t run = 0;
#pragma unroll
                for (int i = 0; i < NB / 32; ++i) {
                    v[i] = run;
                    run += sm.hist[tid * (NB / 32) + i];
                }
                uint32_t inc = run;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const uint32_t o = __shfl_up_sync(0xFFFFFFFFu, inc, d);
                    if (tid >= d) inc += o;
                }
                const uint32_t ex = inc - run;
#pragma unroll
                for (int i = 0; i < NB / 32; ++i) sm.loc[tid * (NB / 32) + i] = ex + v[i];
            }
            if (claimer) next_tile(&sm.tile[turn ^ 1]);
            __syncthreads();
#pragma unroll
            for (int r = 0; r < IPT; ++r) {
                const uint32_t b = (br[r] & 0x7FFu) >> 2;
                if (b < (uint32_t)NB) {
                    const uint32_t p = sm.loc[b] + (br[r] >> 11);
                    sm.u.c.stage[p] = key[r];
                    sm.u.c.bkt[p] = (uint8_t)b;
                }
            }
            if (tid < NB) {
                sm.w.ptr[tid] = reinterpret_cast<uint64_t>(
                    a.out + (overflows() ? a.junk : sm.out_base + sm.region_off[tid] + off) - sm.loc[tid]);
                sm.hist[tid] = 0;
            }
            advance();
            __syncthreads();
            for (uint32_t i = tid; i < tile_cnt; i += THREADS)
                reinterpret_cast<K*>(sm.w.ptr[sm.u.c.bkt[i]])[i] = sm.u.c.stage[i];
        }
    }
}

// Testing: shrink every bucket capacity of segment 0 (forces an overflow).
template <typename K>
__global__ void inject_overflow_kernel(SplitSet<K>* splits, LearnedSet<K>* learned) {
    const int b = threadIdx.x;
    if (b < NB) {
        if (splits[0].region_cap[b] > 16) splits[0].region_cap[b] = 16;
        if (learned && learned[0].region_cap[b] > 16) learned[0].region_cap[b] = 16;
    }
}

// Testing: reject every learned model of the level.
template <typename K>
__global__ void inject_reject_kernel(LearnedSet<K>* learned, uint32_t nsegs) {
    for (uint32_t s = threadIdx.x; s < nsegs; s += blockDim.x) learned[s].ok = 0;
}

// Exact histogram of a level (the fallback after a capacity overflow).
template <typename K, typename InCodec, int THREADS, int IPT>
__global__ void __launch_bounds__(THREADS) count_kernel(PartArgs<K> a, InCodec in) {
    __shared__ K tree[NB];
    __shared__ K uniq[NB];
    __shared__ uint8_t range_b[NB], eq_b[NB];
    __shared__ uint32_t eq_mask[NB / 32];
    __shared__ uint32_t hist[NB];
    __shared__ uint32_t has_eq;
    constexpr int TILE = THREADS * IPT;
    const uint32_t ntiles = a.ntiles_dev ? *a.ntiles_dev : a.ntiles;
    for (uint32_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const uint32_t seg = a.tile_seg ? a.tile_seg[t] : 0u;
        const SegDesc sd = a.segs[seg];
        const SplitSet<K>& ss = a.splits[seg];
        for (int b = threadIdx.x; b < NB; b += THREADS) {
            tree[b] = ss.tree[b];
            uniq[b] = ss.uniq[b];
            range_b[b] = ss.range_b[b];
            eq_b[b] = ss.eq_b[b];
            hist[b] = 0;
        }
        if (threadIdx.x < NB / 32) eq_mask[threadIdx.x] = ss.eq_mask[threadIdx.x];
        if (threadIdx.x == 0) has_eq = ss.has_eq;
        __syncthreads();
        const uint32_t ti = t - sd.tile_start;
        const uint64_t base = sd.in_off + (uint64_t)ti * TILE;
        const uint64_t rem = sd.count - (uint64_t)ti * TILE;
        const uint32_t cnt = rem < (uint64_t)TILE ? (uint32_t)rem : (uint32_t)TILE;
        for (uint32_t i = threadIdx.x; i < cnt; i += THREADS) {
            const K x = in.load(base + i);
            atomicAdd(&hist[find_bucket<K>(tree, x, has_eq != 0, uniq, range_b, eq_b, eq_mask)], 1u);
        }
        __syncthreads();
        for (int b = threadIdx.x; b < NB; b += THREADS)
            if (hist[b]) atomicAdd(&a.fill[(size_t)seg * NB + b], (unsigned long long)hist[b]);
        __syncthreads();
    }
}

// Re-lay the bucket regions of every segment from exact counts.
template <typename K>
__global__ void __launch_bounds__(NB) exact_regions_kernel(SplitSet<K>* splits, const uint64_t* bucket_counts,
                                                           uint32_t nsegs) {
    __shared__ uint64_t wtot64[8];
    const uint32_t s = blockIdx.x;
    if (s >= nsegs) return;
    const uint64_t c = bucket_counts[(size_t)s * NB + threadIdx.x];
    const uint64_t cap = (c + 15) & ~15ull;
    const uint64_t off = block_exclusive_scan_first<NB, uint64_t>(cap, wtot64, (uint64_t*)nullptr);
    splits[s].region_off[threadIdx.x] = off;
    splits[s].region_cap[threadIdx.x] = cap;
}

// ===========================================================================
// 5. Planning: classify each bucket of each segment (one block per segment)

template <typename K>
struct PlanArgs {
    const SegDesc* segs;
    const SplitSet<K>* splits;
    const LearnedSet<K>* learned;       // used for segments whose model was accepted
    const uint64_t* bucket_counts;
    const K* level_out;                 // the level's output buffer
    LeafItem<K>* items[NCLASS + 1];     // per class, plus the copy list
    uint32_t item_cap;
    SegDesc* next;                      // next-level segments (in_off into level_out)
    uint32_t next_cap;
    LevelCtl* ctl;
    int key_bytes;
};

template <typename K>
__global__ void __launch_bounds__(NB) plan_kernel(PlanArgs<K> a, uint32_t nsegs) {
    __shared__ uint64_t wtot64[8];
    const uint32_t s = blockIdx.x;
    if (s >= nsegs) return;
    // (a pass that reported an error leaves no work: leaves may already be
    // queued behind this launch)
    if (a.ctl->err & (DEV_ERR_OVERFLOW | DEV_ERR_TIMEOUT)) return;
    const SegDesc sd = a.segs[s];
    const bool use_learned = a.learned && a.learned[s].ok;
    const uint32_t nbk = use_learned ? a.learned[s].nbuckets : a.splits[s].nbuckets;
    const uint64_t* region_off = use_learned ? a.learned[s].region_off : a.splits[s].region_off;
    const uint32_t* bucket_eq = use_learned ? a.learned[s].bucket_eq : a.splits[s].bucket_eq;
    const int b = threadIdx.x;
    if (b == 0) {
        atomicAdd(use_learned ? &a.ctl->learned_used : &a.ctl->plain_used, 1u);
        if (a.learned && a.learned[s].fitted) {
            atomicAdd(&a.ctl->learned_fitted, 1u);
            atomicMax(&a.ctl->model_imb_bits, __float_as_uint(a.learned[s].max_over_mean));  // (>= 0)
        }
    }
    const uint64_t c = (b < (int)nbk) ? a.bucket_counts[(size_t)s * NB + b] : 0ull;
    const uint64_t excl = block_exclusive_scan_first<NB, uint64_t>(c, wtot64, (uint64_t*)nullptr);
    // what the bucket becomes: a copy (equality bucket or single key, in
    // chunks), a leaf of some class, or a segment of the next level
    constexpr int LIST_NEXT = NCLASS + 1;  // lists 0..NCLASS-1 leaves, NCLASS copies, NCLASS+1 next level
    __shared__ uint32_t list_n[NCLASS + 2], list_base[NCLASS + 2];
    __shared__ uint32_t st_max, st_nonempty;
    __shared__ unsigned long long st_keys, st_next_keys;
    __shared__ double st_sq;
    if (b < NCLASS + 2) list_n[b] = 0;
    if (b == 0) {
        st_max = 0;
        st_nonempty = 0;
        st_keys = 0;
        st_next_keys = 0;
        st_sq = 0.0;
    }
    __syncthreads();
    const bool is_eq = (bucket_eq[b >> 5] >> (b & 31)) & 1u;
    int list = -1;
    uint32_t nslots = 0;
    if (c > 0) {
        if (is_eq || c == 1) {
            list = CLS_COPY;
            nslots = (uint32_t)((c + COPY_CHUNK - 1) / COPY_CHUNK);
        } else if (c <= leaf_max(a.key_bytes)) {
            list = class_of(a.key_bytes, (uint32_t)c);
            nslots = 1;
        } else {
            list = LIST_NEXT;
            nslots = 1;
        }
    }
    // the level's statistics and the list slots, gathered in the block: one
    // global atomic per block and counter instead of one per bucket
    const uint32_t local = list >= 0 ? atomicAdd(&list_n[list], nslots) : 0u;
    {
        uint32_t mx = (uint32_t)(c > 0xFFFFFFFFull ? 0xFFFFFFFFull : c), ne = c > 0 ? 1u : 0u;
        unsigned long long keys = c, nk = list == LIST_NEXT ? c : 0ull;
        double sq = (double)c * (double)c;
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
            mx = max(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, d));
            ne += __shfl_xor_sync(0xFFFFFFFFu, ne, d);
            keys += __shfl_xor_sync(0xFFFFFFFFu, keys, d);
            nk += __shfl_xor_sync(0xFFFFFFFFu, nk, d);
            sq += __shfl_xor_sync(0xFFFFFFFFu, sq, d);
        }
        if ((b & 31) == 0 && ne) {
            atomicMax(&st_max, mx);
            atomicAdd(&st_nonempty, ne);
            atomicAdd(&st_keys, keys);
            atomicAdd(&st_next_keys, nk);
            atomicAdd(&st_sq, sq);
        }
    }
    __syncthreads();
    if (b < NCLASS + 2 && list_n[b]) {
        unsigned int* ctr = b == LIST_NEXT ? &a.ctl->n_next : &a.ctl->n_items[b];
        list_base[b] = atomicAdd(ctr, list_n[b]);
    }
    if (b == 0 && st_nonempty) {
        atomicMax(&a.ctl->max_bucket, st_max);
        atomicAdd(&a.ctl->nonempty, st_nonempty);
        atomicAdd((unsigned long long*)&a.ctl->level_keys, st_keys);
        atomicAdd(&a.ctl->bucket_sq, st_sq);
        if (st_next_keys) atomicAdd((unsigned long long*)&a.ctl->next_keys, st_next_keys);
    }
    __syncthreads();
    if (list < 0) return;
    const K* src = a.level_out + sd.out_base + region_off[b];
    const uint64_t dst = sd.final_off + excl;
    const uint32_t first = list_base[list] + local;
    if (list == CLS_COPY) {
        uint32_t slot = first;
        for (uint64_t o = 0; o < c; o += COPY_CHUNK, ++slot) {
            if (slot < a.item_cap) {
                LeafItem<K> it;
                it.src = src + o;
                it.dst = dst + o;
                it.count = (uint32_t)((c - o) < COPY_CHUNK ? (c - o) : COPY_CHUNK);
                it.pad_ = 0;
                a.items[CLS_COPY][slot] = it;
            } else {
                raise_error(&a.ctl->err, DEV_ERR_CAPACITY);
            }
        }
    } else if (list < NCLASS) {
        if (first < a.item_cap) {
            LeafItem<K> it;
            it.src = src;
            it.dst = dst;
            it.count = (uint32_t)c;
            it.pad_ = 0;
            a.items[list][first] = it;
        } else {
            raise_error(&a.ctl->err, DEV_ERR_CAPACITY);
        }
    } else {
        if (first < a.next_cap) {
            SegDesc n;
            n.in_off = sd.out_base + region_off[b];
            n.count = c;
            n.final_off = dst;
            n.out_base = 0;
            n.tile_start = 0;
            n.ntiles = 0;
            a.next[first] = n;
        } else {
            raise_error(&a.ctl->err, DEV_ERR_CAPACITY);
        }
    }
}

// Give the next level's segments their tiles and output regions (one block).
static __global__ void __launch_bounds__(1024) prepare_level_kernel(SegDesc* segs, uint32_t nsegs, uint32_t tile,
                                                             LevelCtl* ctl_next) {
    __shared__ uint64_t wt1[32], wt2[32];
    __shared__ uint64_t tot1, tot2;
    __shared__ uint64_t carry_tiles, carry_bound;
    if (threadIdx.x == 0) {
        carry_tiles = 0;
        carry_bound = 0;
    }
    __syncthreads();
    for (uint32_t base = 0; base < nsegs; base += 1024) {
        const uint32_t s = base + threadIdx.x;
        uint64_t nt = 0, bd = 0;
        if (s < nsegs) {
            nt = (segs[s].count + tile - 1) / tile;
            bd = (region_bound(segs[s].count) + 15) & ~15ull;
        }
        const uint64_t ex_t = block_exclusive_scan_first<1024, uint64_t>(nt, wt1, &tot1);
        const uint64_t ex_b = block_exclusive_scan_first<1024, uint64_t>(bd, wt2, &tot2);
        if (s < nsegs) {
            segs[s].tile_start = (uint32_t)(carry_tiles + ex_t);
            segs[s].ntiles = (uint32_t)nt;
            segs[s].out_base = carry_bound + ex_b;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            carry_tiles += tot1;
            carry_bound += tot2;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        ctl_next->ntiles_next = (uint32_t)carry_tiles;
        ctl_next->bound_next = carry_bound;
    }
}

// tile -> segment map (one block per segment)
static __global__ void tile_map_kernel(const SegDesc* segs, uint32_t nsegs, uint32_t* tile_seg) {
    const uint32_t s = blockIdx.x;
    if (s >= nsegs) return;
    const SegDesc sd = segs[s];
    for (uint32_t i = threadIdx.x; i < sd.ntiles; i += blockDim.x) tile_seg[sd.tile_start + i] = s;
}

// ===========================================================================
// 6. Leaves

// One warp per bucket of at most 32*IPT keys (class 0).
template <typename K, typename OutCodec, int IPT>
__global__ void __launch_bounds__(256) leaf_warp_kernel(const LeafItem<K>* __restrict__ items, uint32_t nitems,
                                                        OutCodec out) {
    __shared__ K stage[8][32 * IPT];
    const unsigned warp = threadIdx.x >> 5, lane = lane_id();
    K* sw = stage[warp];
    for (uint32_t it = blockIdx.x * 8 + warp; it < nitems; it += gridDim.x * 8) {
        const LeafItem<K> item = items[it];
        for (uint32_t i = lane; i < 32 * IPT; i += 32) sw[i] = i < item.count ? item.src[i] : KeyMax<K>::value;
        __syncwarp();
        K x[IPT];
#pragma unroll
        for (int r = 0; r < IPT; ++r) x[r] = sw[lane * IPT + r];
        __syncwarp();
        warp_bitonic_sort<K, IPT>(x);
#pragma unroll
        for (int r = 0; r < IPT; ++r) sw[lane * IPT + r] = x[r];
        __syncwarp();
        for (uint32_t i = lane; i < item.count; i += 32) out.store(item.dst + i, sw[i]);
        __syncwarp();
    }
}

// Blocks per SM that the leaf kernel's register budget is sized for.  (The
// 4608-key class, which holds most buckets of a large sort, has 12 keys per
// thread: 36 warps an SM instead of 27 with 288 threads of 16, 1.07 -> 1.03 ms
// of 2^28 doubles.)
__host__ __device__ constexpr int leaf_min_blocks(int threads) {
    return (threads == 288 || threads == 320 || threads == 384) ? 3 : 1024 / threads;
}

// One block per bucket of at most THREADS*EPT keys: distribution counting
// into value slots (s512_slotsort.cuh).  The next bucket's keys are loaded
// into registers while the current one is ranked and written.  A bucket whose
// slots come out uneven is appended to `uneven` (count in *n_uneven) for
// leaf_uneven_kernel.
template <typename K, typename OutCodec, int THREADS, int EPT>
__global__ void __launch_bounds__(THREADS, leaf_min_blocks(THREADS))
    leaf_block_kernel(const LeafItem<K>* __restrict__ items, uint32_t nitems, OutCodec out, LeafItem<K>* uneven,
                      uint32_t* n_uneven) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ SlotRed<K> red;
    uint32_t it = blockIdx.x;
    if (it >= nitems) return;
    LeafItem<K> cur = items[it];
    K key[EPT];
    auto load = [&](const LeafItem<K>& item) {
#pragma unroll
        for (int r = 0; r < EPT; ++r) {
            const uint32_t i = (uint32_t)r * THREADS + threadIdx.x;
            if (i < item.count) key[r] = __ldg(item.src + i);
        }
    };
    load(cur);
    for (; it < nitems; it += gridDim.x) {
        const uint32_t nx = it + gridDim.x;
        LeafItem<K> next;
        next.count = 0;
        if (nx < nitems) next = items[nx];
        const size_t dst = cur.dst;
        block_slot_sort<K, THREADS, EPT, SLOT_HAND>(
            key, cur.count, [&](uint32_t i, K x) { out.store(dst + i, x); }, [&]() { load(next); },
            [&]() { uneven[atomicAdd(n_uneven, 1u)] = cur; }, smem_raw, red);
        cur = next;
    }
}

// Every bucket of up to ANY_CAP keys of a level, and its copies, in one launch
// that reads the counts on the device: it is queued behind the plan before the
// host has seen them, and one size of block sorts all classes.  Its last block
// writes the control block to the host's page-locked copy (a copy of its own
// behind it: 6 us).  For levels of
// few keys, where a read-back and a launch per class cost more than blocks
// that fit their buckets save (2^20 int32: eight leaf launches and their gaps
// 45 us, this one 9 us).  The host launches what it leaves: larger
// buckets, and those found uneven.
constexpr int ANY_THREADS = 512;
constexpr int ANY_CLASSES = 8;  // leaf classes 0..7
constexpr int ANY_CAP = class_cap(ANY_CLASSES - 1);
static_assert(ANY_CAP == ANY_THREADS * 16, "the largest class fills a block's 16 keys per thread");
template <typename K>
struct LeafLists {
    const LeafItem<K>* items;  // NCLASS + 1 lists of `cap` items each
    uint32_t cap;
};
template <typename K, typename OutCodec>
__global__ void __launch_bounds__(ANY_THREADS, 2) leaf_any_kernel(LeafLists<K> lists, LevelCtl* ctl, OutCodec out,
                                                                  LeafItem<K>* uneven, LevelCtl* host_ctl) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ SlotRed<K> red;
    __shared__ uint32_t last;
    uint32_t total = ctl->n_items[CLS_COPY];
#pragma unroll
    for (int c = 0; c < ANY_CLASSES; ++c) total += ctl->n_items[c];
    if (ctl->err) total = 0;  // (the host redoes the level, or reports the error)
    for (uint32_t it = blockIdx.x; it < total; it += gridDim.x) {
        uint32_t i = it;
        int c = ANY_CLASSES - 1;  // the largest first, the copies last
        for (; c >= 0; --c) {
            const uint32_t n = ctl->n_items[c];
            if (i < n) break;
            i -= n;
        }
        const LeafItem<K> item = lists.items[(size_t)(c < 0 ? CLS_COPY : c) * lists.cap + i];
        auto store = [&](uint32_t k, K x) { out.store(item.dst + k, x); };
        auto give = [&]() { uneven[atomicAdd(&ctl->n_uneven[ANY_CLASSES - 1], 1u)] = item; };
        auto sort = [&](auto ept) {
            constexpr int EPT = decltype(ept)::value;
            K key[EPT];
#pragma unroll
            for (int r = 0; r < EPT; ++r) {
                const uint32_t k = (uint32_t)r * ANY_THREADS + threadIdx.x;
                if (k < item.count) key[r] = __ldg(item.src + k);
            }
            block_slot_sort<K, ANY_THREADS, EPT, SLOT_HAND>(key, item.count, store, [] {}, give, smem_raw, red);
        };
        if (c < 0) {
            for (uint32_t k = threadIdx.x; k < item.count; k += ANY_THREADS) store(k, item.src[k]);
        } else if (item.count > ANY_THREADS * 8) {
            sort(std::integral_constant<int, 16>{});
        } else {
            sort(std::integral_constant<int, 8>{});
        }
        __syncthreads();  // (the two sizes lay out shared memory differently)
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(&ctl->blocks_done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (last) {
        __threadfence();
        for (uint32_t i = threadIdx.x; i < sizeof(LevelCtl) / 4; i += ANY_THREADS)
            reinterpret_cast<volatile uint32_t*>(host_ctl)[i] = reinterpret_cast<volatile uint32_t*>(ctl)[i];
    }
}

// Which leaves that came out uneven are dealt a second time before the block
// sort.  Not key/value pairs (see block_slot_sort on `refine`), nor the leaves
// of 32-bit arrays: they are uneven because values repeat, several to a coarse
// slot (2^27 Zipf int32: 3.09 ms a sort with the second dealing, 2.84 without).
template <typename K, typename OutCodec>
constexpr bool leaf_refines() { return !OutCodec::PAIRS && sizeof(K) == 8; }

// The buckets the slot sort found uneven: refined slots where leaf_refines, else
// (and where those are uneven too) bitonic leaves + merge path.
template <typename K, typename OutCodec, int THREADS, int EPT>
__global__ void __launch_bounds__(THREADS, !leaf_refines<K, OutCodec>() || 1024 / THREADS < 2 ? 1024 / THREADS : 2)
    leaf_uneven_kernel(const LeafItem<K>* __restrict__ items, const uint32_t* n_items, OutCodec out) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const uint32_t nitems = *n_items;
    for (uint32_t it = blockIdx.x; it < nitems; it += gridDim.x) {
        const LeafItem<K> item = items[it];
        if constexpr (!leaf_refines<K, OutCodec>()) {
            K* s = reinterpret_cast<K*>(smem_raw);
            for (uint32_t i = threadIdx.x; i < item.count; i += THREADS) s[pidx(i)] = item.src[i];
            block_merge_sort<K, THREADS, EPT>(s, item.count);
            for (uint32_t i = threadIdx.x; i < item.count; i += THREADS) out.store(item.dst + i, s[pidx(i)]);
        } else {
            __shared__ SlotRed<K> red;
            K key[EPT];
#pragma unroll
            for (int r = 0; r < EPT; ++r) {
                const uint32_t i = (uint32_t)r * THREADS + threadIdx.x;
                if (i < item.count) key[r] = __ldg(item.src + i);
            }
            block_slot_sort<K, THREADS, EPT, SLOT_REFINE>(
                key, item.count, [&](uint32_t i, K x) { out.store(item.dst + i, x); }, [] {}, [] {}, smem_raw, red);
        }
        __syncthreads();  // (the next bucket's keys go where other threads may still read these)
    }
}
template <typename K, typename OutCodec, int THREADS, int EPT>
constexpr size_t leaf_uneven_smem() {
    using SM = SlotSmem<K, THREADS, EPT>;
    return leaf_refines<K, OutCodec>() ? SM::bytes : SM::padded_bytes;
}

// Copy equality buckets (and single keys) to their final place.
template <typename K, typename OutCodec>
__global__ void __launch_bounds__(256) leaf_copy_kernel(const LeafItem<K>* __restrict__ items, uint32_t nitems,
                                                        OutCodec out) {
    for (uint32_t it = blockIdx.x; it < nitems; it += gridDim.x) {
        const LeafItem<K> item = items[it];
        for (uint32_t i = threadIdx.x; i < item.count; i += 256) out.store(item.dst + i, item.src[i]);
    }
}

// ===========================================================================
// 7. Whole arrays that fit one leaf: sort straight from and to the caller's layout.

template <typename InCodec, typename OutCodec, int IPT>
__global__ void __launch_bounds__(32) small_warp_sort_kernel(InCodec in, OutCodec out, uint32_t n) {
    using K = typename InCodec::Key;
    __shared__ K sw[32 * IPT];
    const unsigned lane = lane_id();
    for (uint32_t i = lane; i < 32 * IPT; i += 32) sw[i] = i < n ? in.load(i) : KeyMax<K>::value;
    __syncwarp();
    K x[IPT];
#pragma unroll
    for (int r = 0; r < IPT; ++r) x[r] = sw[lane * IPT + r];
    __syncwarp();
    warp_bitonic_sort<K, IPT>(x);
#pragma unroll
    for (int r = 0; r < IPT; ++r) sw[lane * IPT + r] = x[r];
    __syncwarp();
    for (uint32_t i = lane; i < n; i += 32) out.store(i, sw[i]);
}

template <typename InCodec, typename OutCodec, int THREADS, int EPT>
__global__ void __launch_bounds__(THREADS, 1024 / THREADS) small_block_sort_kernel(InCodec in, OutCodec out,
                                                                                   uint32_t n) {
    using K = typename InCodec::Key;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ SlotRed<K> red;
    K key[EPT];
#pragma unroll
    for (int r = 0; r < EPT; ++r) {
        const uint32_t i = (uint32_t)r * THREADS + threadIdx.x;
        if (i < n) key[r] = in.load(i);
    }
    block_slot_sort<K, THREADS, EPT, SLOT_INLINE>(
        key, n, [&](uint32_t i, K x) { out.store(i, x); }, [] {}, [] {}, smem_raw, red, !OutCodec::PAIRS);
}
}  // namespace s512
