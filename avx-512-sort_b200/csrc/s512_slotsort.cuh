// s512_slotsort.cuh -- one bucket sorted by distribution counting: keys are
// dealt into value slots by a monotone linear map of their offset from the
// bucket's minimum, the slots are laid out by an exclusive scan of their
// counts, the keys are dealt into their slots, and each slot that received
// more than one key (a few keys at most) is put in order in place by one
// thread; the buffer is then the sorted bucket.
//
// A bucket that reaches the leaf stage holds the keys between two adjacent
// quantile splitters, so its values are close to evenly spread over
// [min, max]: with four slots per key of the class, four keys in five have a
// slot of their own and the whole sort costs a few shared-memory operations
// per key, where a comparison network costs one compare-exchange per key for
// every stage.  When the spread is uneven (a cluster, a run of repeated
// values, an outlier that stretches the range) the slot counts show it before
// any key moves: if a slot holds more than SLOT_MAX keys, or some thread's
// keys met more than SLOT_MEET others each on average, the bucket is dealt
// again through slots refined by the first counts (refine_slots), and by the
// bitonic + merge-path block sort (s512_blocksort.cuh) if those are uneven too.
//
// What bounds it: issue slots and shared-memory latency, not HBM, so the code
// is laid out for few instructions per key.  Four 8-bit slot counters share a
// word: one atomic gives a key its rank in its slot, and the scan leaves in
// the same word the first key's place (14 bits) and the running counts of the
// word's first three slots (6 bits each), so a key finds its place with one
// more load.  Measured: the leaves of 2^28 uniform doubles 2.46 -> 1.99 ms
// against one 32-bit counter per key, a second atomic to deal it and 64-bit
// bounds; one array of 10007 uniform doubles, whose bit patterns crowd into
// the top binade, 48 -> 15 us, because four slots per key keep it out of the
// block sort.
//
// Equal keys are identical encoded words (see s512_common.cuh), so placing
// ties in any order gives the same output.
#pragma once

#include "s512_blocksort.cuh"

namespace s512 {

constexpr uint32_t SLOT_MAX = 16;   // largest slot put in order by one thread (3 * 16 < 64: the
                                    // running counts of a word fit their 6 bits)
constexpr uint32_t SLOT_MEET = 3;   // a thread's keys may meet this many earlier keys each, on average

// Monotone map from a key in [lo, hi] to a slot in [0, nslots): the offset
// x - lo is cut to its 32 leading significant bits (shift sh), then either
// used as the slot itself (direct, when the cut range is below nslots) or
// scaled by mul / 2^32 with mul just below nslots * 2^32 / (range + 1), which
// keeps the largest offset below nslots.
template <typename K>
struct SlotMap {
    K lo;
    uint32_t sh, mul, direct;
    __device__ __forceinline__ uint32_t operator()(K x) const {
        uint32_t d;
        if constexpr (sizeof(K) == 8) d = (uint32_t)((x - lo) >> sh);
        else d = (uint32_t)(x - lo);  // (32-bit offsets need no shift)
        return direct ? d : __umulhi(d, mul);
    }
};

// The slot map of [lo, lo + range].  The quotient is taken in float, rounded
// down far enough that the largest offset stays below nslots (a 64-bit
// division costs as much as seven keys of work).
template <typename K>
__device__ __forceinline__ SlotMap<K> make_slot_map(K lo, K range, uint32_t nslots) {
    SlotMap<K> f;
    f.lo = lo;
    int nb;
    if constexpr (sizeof(K) == 8) nb = 64 - __clzll((long long)range);
    else nb = 32 - __clz((int)range);
    f.sh = nb > 32 ? (uint32_t)(nb - 32) : 0u;
    const uint32_t dr = (uint32_t)(range >> f.sh);
    f.direct = dr < nslots ? 1u : 0u;
    // relative error of the conversion, the divide and the product: under
    // 2^-21; the factor takes off 2^-20
    const float q = __fdividef((float)nslots * 4294967296.0f, (float)dr + 1.0f) * (1.0f - 1.0f / 1048576.0f);
    f.mul = f.direct ? 0u : (uint32_t)q;
    return f;
}

enum SlotPath { SLOT_EQUAL, SLOT_EVEN, SLOT_UNEVEN };

// Per-warp partials of the block reductions.
template <typename K>
struct SlotRed {
    K wlo[32], whi[32];
    uint32_t hlo[32], hhi[32];
    uint32_t wtot[32];
};

// Shared memory of block_slot_sort for a block of THREADS x IPT keys: the
// key buffer, one word of four slot counters per key, and the list of the
// slots that received several keys (at most half as many as keys; before that
// list is written its space holds the big slots of refine_slots).  The block
// sort, where it may run (INLINE), lays its padded keys over all of it.
template <typename K, int THREADS, int IPT, bool INLINE = true>
struct SlotSmem {
    static constexpr uint32_t S = (uint32_t)THREADS * IPT;
    static constexpr size_t keys_bytes = (size_t)S * sizeof(K);
    static constexpr size_t ctr_bytes = (size_t)S * sizeof(uint32_t);
    static constexpr size_t list_bytes = (size_t)S;
    static constexpr size_t slot_bytes = keys_bytes + ctr_bytes + list_bytes;
    static constexpr size_t padded_bytes = ((size_t)padded_len(S) * sizeof(K) + 15) & ~(size_t)15;
    static constexpr size_t bytes = INLINE && padded_bytes > slot_bytes ? padded_bytes : slot_bytes;
};

// Byte offset of a counter word in shared memory.  A thread scans IPT
// consecutive words as 16-byte quads; exchanging quads within a thread's
// group keeps the eight lanes of a quad access on different banks (their
// stride would otherwise put them four or two to a bank; at IPT 12 the stride
// does it by itself).  The exchange is its own inverse.
template <int IPT>
__device__ __forceinline__ uint32_t ctr_swizzle(uint32_t a) {
    constexpr uint32_t Q = IPT / 4;
    if constexpr (Q == 2 || Q == 4) return a ^ ((a >> 3) & ((Q - 1) << 4));
    else return a;
}

// How many of the c keys held striped in key[] this thread holds (key[r] is
// one for r below that: a compare with a constant per key and phase).
template <int THREADS>
__device__ __forceinline__ int own_keys(uint32_t c) {
    return threadIdx.x < c ? (int)((c - threadIdx.x + THREADS - 1) / THREADS) : 0;
}

// Bounds of the c keys held striped in key[]: lo <= every key <= lo + range.
// Of 64-bit keys only the high words are compared: unless they span very few
// values, the bounds need no more precision (range == 0 is always exact).
// Every thread of the block calls it; it has a barrier.
template <typename K, int THREADS, int IPT>
__device__ __forceinline__ void block_bounds(const K (&key)[IPT], uint32_t c, SlotRed<K>& red, K& lo, K& range) {
    constexpr int NW = THREADS / 32;
    const unsigned tid = threadIdx.x, lane = lane_id(), warp = tid >> 5;
    const int own = own_keys<THREADS>(c);
    uint32_t hmin = 0xFFFFFFFFu, hmax = 0u;
#pragma unroll
    for (int r = 0; r < IPT; ++r) {
        if (r < own) {
            const uint32_t h = sizeof(K) == 8 ? (uint32_t)((uint64_t)key[r] >> 32) : (uint32_t)key[r];
            hmin = min(hmin, h);
            hmax = max(hmax, h);
        }
    }
    hmin = __reduce_min_sync(0xFFFFFFFFu, hmin);
    hmax = __reduce_max_sync(0xFFFFFFFFu, hmax);
    if (lane == 0) {
        red.hlo[warp] = hmin;
        red.hhi[warp] = hmax;
    }
    __syncthreads();
    hmin = __reduce_min_sync(0xFFFFFFFFu, lane < (unsigned)NW ? red.hlo[lane] : 0xFFFFFFFFu);
    hmax = __reduce_max_sync(0xFFFFFFFFu, lane < (unsigned)NW ? red.hhi[lane] : 0u);
    if constexpr (sizeof(K) == 8) {
        lo = (uint64_t)hmin << 32;
        range = ((uint64_t)(hmax - hmin) << 32) | 0xFFFFFFFFull;
        if (hmax - hmin < 4096u) {  // few high words: exact bounds
            K mn = KeyMax<K>::value, mx = K(0);
#pragma unroll
            for (int r = 0; r < IPT; ++r) {
                if (r < own) {
                    mn = kmin(mn, key[r]);
                    mx = kmax(mx, key[r]);
                }
            }
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) {
                mn = kmin(mn, shfl_xor(mn, d));
                mx = kmax(mx, shfl_xor(mx, d));
            }
            if (lane == 0) {
                red.wlo[warp] = mn;
                red.whi[warp] = mx;
            }
            __syncthreads();
            mn = lane < (unsigned)NW ? red.wlo[lane] : KeyMax<K>::value;
            mx = lane < (unsigned)NW ? red.whi[lane] : K(0);
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) {
                mn = kmin(mn, shfl_xor(mn, d));
                mx = kmax(mx, shfl_xor(mx, d));
            }
            lo = mn;
            range = mx - mn;
        }
    } else {
        lo = hmin;
        range = hmax - hmin;
    }
}

enum SlotMode { SLOT_HAND, SLOT_INLINE, SLOT_REFINE };

// A coarse slot of more than SLOT_MAX keys: its keys' own bounds, as a map to
// four fine slots per key.
template <typename K>
struct alignas(16) BigSlot {
    K lo;
    uint32_t mul;   // (the slot's count until its bounds are known)
    uint32_t aux;   // first place | shift << 16 | direct << 22 | all equal << 23 | one value << 24
};

// Fine slots for a bucket whose values crowd: every key's slot of 4*c, rising
// with the keys, into fine[].  The bucket is dealt once into as many coarse
// slots as the class has keys; the keys of a coarse slot then spread over four
// fine slots per key, by their place between the slot's own lowest and highest
// key where it holds many (a cluster, a hot key's values: exact bounds, found
// by a warp from the dealt keys; equal keys by their rank, so that any number
// of them fits, also between a few other keys), by their place in the slot
// where it holds few.
// Leaves the counters zeroed, a barrier behind.
template <typename K, int THREADS, int IPT>
__device__ __forceinline__ void refine_slots(const K (&key)[IPT], uint32_t c, K lo, K range, uint32_t (&fine)[IPT],
                                             K* s, unsigned char* ctr, BigSlot<K>* big, SlotRed<K>& red) {
    constexpr uint32_t S = (uint32_t)THREADS * IPT;
    constexpr int NW = THREADS / 32;
    constexpr uint32_t BIG = 0x80000000u;
    const unsigned tid = threadIdx.x, lane = lane_id(), warp = tid >> 5;
    auto zero = [&]() {
#pragma unroll
        for (int r = 0; r < IPT; r += 4)
            *reinterpret_cast<uint4*>(ctr + (size_t)tid * IPT * 4 + r * 4) = make_uint4(0u, 0u, 0u, 0u);
    };
    auto quad = [&](int j) {
        return reinterpret_cast<uint4*>(ctr + ctr_swizzle<IPT>(tid * IPT * 4 + (uint32_t)j * 16));
    };
    zero();
    __syncthreads();
    // coarse counts; a key's rank in its slot
    const SlotMap<K> f = make_slot_map<K>(lo, range, S);
#pragma unroll
    for (int r = 0; r < IPT; ++r) {
        if ((uint32_t)r * THREADS + tid < c) {
            const uint32_t a = ctr_swizzle<IPT>(f(key[r]) * 4u);
            fine[r] = a | (atomicAdd(reinterpret_cast<uint32_t*>(ctr + a), 1u) << 16);  // (both under 2^16)
        }
    }
    __syncthreads();
    // places (low half) and numbers of big slots (high half) before each word
    uint32_t v = 0;
#pragma unroll
    for (int j = 0; j < IPT / 4; ++j) {
        const uint4 q = *quad(j);
        v += q.x + q.y + q.z + q.w;
        v += ((q.x > SLOT_MAX ? 1u : 0u) + (q.y > SLOT_MAX ? 1u : 0u) + (q.z > SLOT_MAX ? 1u : 0u) +
              (q.w > SLOT_MAX ? 1u : 0u)) << 16;
    }
    uint32_t inc = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t o = __shfl_up_sync(0xFFFFFFFFu, inc, d);
        if (lane >= (unsigned)d) inc += o;
    }
    if (lane == 31) red.wtot[warp] = inc;
    __syncthreads();
    const uint32_t wt = lane < (unsigned)NW ? red.wtot[lane] : 0u;
    uint32_t run = __reduce_add_sync(0xFFFFFFFFu, lane < warp ? wt : 0u) + inc - v;
    const uint32_t nbig = __reduce_add_sync(0xFFFFFFFFu, wt) >> 16;  // (at most S / 16)
#pragma unroll
    for (int j = 0; j < IPT / 4; ++j) {
        uint4* qp = quad(j);
        uint4 q = *qp;
        auto word = [&](uint32_t n) {  // first place (14 bits), then the count or the big slot's number
            const uint32_t at = run & 0xFFFFu, id = run >> 16;
            uint32_t w = (at & 0x3FFFu) | (n << 14);  // (5 bits)
            run += n;
            if (n > SLOT_MAX) {
                big[id].mul = n;
                big[id].aux = at;
                w = BIG | (at & 0x3FFFu) | (id << 14);
                run += 1u << 16;
            }
            return w;
        };
        q.x = word(q.x);
        q.y = word(q.y);
        q.z = word(q.z);
        q.w = word(q.w);
        *qp = q;
    }
    __syncthreads();
    // deal into the coarse slots; keep what a key needs of its slot
#pragma unroll
    for (int r = 0; r < IPT; ++r) {
        if ((uint32_t)r * THREADS + tid < c) {
            const uint32_t w = *reinterpret_cast<const uint32_t*>(ctr + (fine[r] & 0xFFFFu));
            const uint32_t rank = fine[r] >> 16;
            s[(w & 0x3FFFu) + rank] = key[r];
            fine[r] = (w & BIG) ? (w & ~0x3FFFu) | rank : w;
        }
    }
    __syncthreads();
    zero();
    for (uint32_t id = warp; id < nbig; id += NW) {
        const uint32_t n = big[id].mul, at = big[id].aux;
        K mn = KeyMax<K>::value, mx = K(0);
#pragma unroll 4
        for (uint32_t i = lane; i < n; i += 32) {
            const K x = s[at + i];
            mn = kmin(mn, x);
            mx = kmax(mx, x);
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
            mn = kmin(mn, shfl_xor(mn, d));
            mx = kmax(mx, shfl_xor(mx, d));
        }
        const SlotMap<K> g = make_slot_map<K>(mn, mx - mn, 4 * n);
        // mostly one value (a quarter of 32 of the keys)?  Then it takes the
        // fine slots, and the others, if few, the first and the last one
        const K x = s[at + lane * n / 32], one = shfl_from(x, 16);
        bool alone = false;
        if (mn != mx && __popc(__ballot_sync(0xFFFFFFFFu, x == one)) >= 8) {
            uint32_t below = 0, above = 0;
            for (uint32_t i = lane; i < n; i += 32) {
                below += s[at + i] < one ? 1u : 0u;
                above += one < s[at + i] ? 1u : 0u;
            }
            below = __reduce_add_sync(0xFFFFFFFFu, below);
            above = __reduce_add_sync(0xFFFFFFFFu, above);
            alone = below <= SLOT_MAX && above <= SLOT_MAX;
        }
        __syncwarp();
        if (lane == 0) {
            BigSlot<K> b;
            b.lo = alone ? one : mn;
            b.mul = alone ? n : g.mul;
            b.aux = at | (g.sh << 16) | (g.direct << 22) | (mn == mx ? 1u << 23 : 0u) | (alone ? 1u << 24 : 0u);
            big[id] = b;
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < IPT; ++r) {
        if ((uint32_t)r * THREADS + tid < c) {
            const uint32_t w = fine[r];
            uint32_t first, sub;
            if (w & BIG) {
                const BigSlot<K> b = big[(w >> 14) & 0x3FFu];
                first = b.aux & 0xFFFFu;
                const uint32_t d = (uint32_t)((key[r] - b.lo) >> ((b.aux >> 16) & 63u));
                const uint32_t by_rank = 4u * (w & 0x3FFFu);
                if (b.aux >> 24)
                    sub = key[r] < b.lo ? 0u
                          : b.lo < key[r] ? 4u * b.mul - 1u
                                          : min(max(by_rank, 1u), 4u * b.mul - 2u);
                else
                    sub = (b.aux >> 23) ? by_rank : (b.aux >> 22) ? d : __umulhi(d, b.mul);
            } else {
                first = w & 0x3FFFu;
                const uint32_t d = (uint32_t)((key[r] - lo) >> f.sh);
                sub = f.direct ? 0u : __umulhi(d * f.mul, 4u * (w >> 14));  // (the fraction of the slot)
            }
            fine[r] = 4u * first + sub;
        }
    }
}

// Sort the c <= THREADS*IPT keys held striped in key[] (element
// r*THREADS + tid in key[r]; entries past c are ignored) into store(0..c).
// `smem` holds SlotSmem<K,THREADS,IPT>::bytes; `red` is the block's reduction
// scratch.  refill() is called exactly once, as soon as key[] is no longer
// needed, so that the caller can start loading the next bucket into it while
// this one is ranked and written.  Every thread of the block must call it.
// The key buffer may still be read by other threads when it returns; another
// call may follow directly (it does not write that buffer before its own
// barriers), anything else needs a barrier first.
// Returns how the bucket was sorted, hence where its sorted keys are left in
// the key buffer: in order (SLOT_EVEN), in the block sort's padded layout
// (SLOT_UNEVEN, where the block sort ran), or nowhere (SLOT_EQUAL).
//
// What happens to an uneven bucket depends on MODE.  SLOT_HAND: thread 0 calls
// uneven() (which hands the bucket to a separate launch) and nothing is
// written; keeping the rest out of the kernel keeps the slot path's register
// budget for the keys.  SLOT_INLINE: it is dealt a second time, through slots
// refined by the first (refine below), and if that leaves it uneven too it is
// sorted by the block sort.  SLOT_REFINE: the same without the first attempt,
// for buckets known to be uneven.  `refine` off leaves the second dealing out:
// words of key/value pairs crowd by hot keys, whose values share their coarse
// slot with a few other keys that stretch its bounds, so refined slots are
// rarely even (2^27 pairs with Zipf keys: uneven leaves 1.11 ms by the block
// sort, 1.54 ms with a second dealing before it).  Doubles gain: a sample of
// 16384 normal doubles (two signs, 60 binades) is sorted in 45 instead of 72 us.
template <typename K, int THREADS, int IPT, SlotMode MODE, typename Store, typename Refill, typename Uneven>
__device__ SlotPath block_slot_sort(K (&key)[IPT], uint32_t c, Store store, Refill refill, Uneven uneven,
                                unsigned char* smem, SlotRed<K>& red, bool refine = true) {
    constexpr uint32_t S = (uint32_t)THREADS * IPT;
    constexpr uint32_t NSLOTS = 4 * S;
    constexpr int NW = THREADS / 32;
    static_assert(IPT % 4 == 0 && IPT <= 16, "counter words are read four at a time");
    static_assert(S <= 16384, "a place is 14 bits, a counter's byte offset 16");
    using SM = SlotSmem<K, THREADS, IPT, MODE != SLOT_HAND>;
    K* s = reinterpret_cast<K*>(smem);
    unsigned char* ctr = smem + SM::keys_bytes;
    uint16_t* list = reinterpret_cast<uint16_t*>(smem + SM::keys_bytes + SM::ctr_bytes);
    const unsigned tid = threadIdx.x, lane = lane_id(), warp = tid >> 5;

    // 1. counters zeroed; bounds of the bucket
#pragma unroll
    for (int r = 0; r < IPT; r += 4)
        *reinterpret_cast<uint4*>(ctr + (size_t)tid * IPT * 4 + r * 4) = make_uint4(0u, 0u, 0u, 0u);
    K lo, range;
    block_bounds<K, THREADS, IPT>(key, c, red, lo, range);
    const int own = own_keys<THREADS>(c);

    if (range == 0) {  // every key equal: already in order
#pragma unroll
        for (int r = 0; r < IPT; ++r) {
            const uint32_t i = (uint32_t)r * THREADS + tid;
            if (i < c) store(i, key[r]);
        }
        refill();
        __syncthreads();  // (the counters and bounds are rewritten by the next call)
        return SLOT_EQUAL;
    }

    // 2. slot counts: a key's rank in its slot is its counter's byte before
    // the key's own increment.  (A byte that passes 255 carries into its
    // neighbour, but then a key has seen a rank of SLOT_MAX or more and the
    // counts are not used.)
    uint32_t pr[IPT];  // counter byte offset | slot within the word | rank << 16
    uint32_t nmulti = 0;
    auto count = [&](uint32_t meet, auto slot_of) {
        uint32_t seen = 0, rsum = 0;
        nmulti = 0;
#pragma unroll
        for (int r = 0; r < IPT; ++r) {
            const uint32_t was = MODE == SLOT_HAND ? 0u : pr[r];
            pr[r] = 0;
            if (r < own) {
                const uint32_t slot = slot_of(r, was);
                const uint32_t a = ctr_swizzle<IPT>(slot & ~3u);
                const uint32_t k8 = slot << 3;  // (shifts take it modulo 32)
                const uint32_t old = atomicAdd(reinterpret_cast<uint32_t*>(ctr + a), __funnelshift_l(0u, 1u, k8));
                const uint32_t rank = __funnelshift_r(old, 0u, k8) & 0xFFu;
                pr[r] = (a | (slot & 3u)) + (rank << 16);
                rsum += rank;
                nmulti += rank == 1u ? 1u : 0u;
            }
            seen |= pr[r];
        }
        static_assert(SLOT_MAX == 16, "a rank of 16 or more sets a bit from the 20th on");
        return !__syncthreads_or((seen >> 20) != 0 || rsum > meet * IPT);
    };
    bool even = false;
    if constexpr (MODE != SLOT_REFINE) {
        const SlotMap<K> f = make_slot_map<K>(lo, range, NSLOTS);
        even = count(SLOT_MEET, [&](int r, uint32_t) { return f(key[r]); });
    }
    if constexpr (MODE != SLOT_HAND) {
        if (!even && refine) {
            refine_slots<K, THREADS, IPT>(key, c, lo, range, pr, s, ctr, reinterpret_cast<BigSlot<K>*>(list), red);
            even = count(2 * SLOT_MEET, [&](int, uint32_t was) { return was; });
        }
    }

    if (even) {
        // 3. exclusive scan of the counts (IPT consecutive words per thread)
        // and, in the high half, of the slots with several keys (each counted
        // by the thread whose key came second)
        uint32_t v = nmulti << 16;
        auto quad = [&](int j) {
            return reinterpret_cast<uint4*>(ctr + ctr_swizzle<IPT>(tid * IPT * 4 + (uint32_t)j * 16));
        };
#pragma unroll
        for (int j = 0; j < IPT / 4; ++j) {
            const uint4 q = *quad(j);
            v = __dp4a(q.x, 0x01010101u, v);
            v = __dp4a(q.y, 0x01010101u, v);
            v = __dp4a(q.z, 0x01010101u, v);
            v = __dp4a(q.w, 0x01010101u, v);
        }
        uint32_t inc = v;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t o = __shfl_up_sync(0xFFFFFFFFu, inc, d);
            if (lane >= (unsigned)d) inc += o;
        }
        if (lane == 31) red.wtot[warp] = inc;
        __syncthreads();
        const uint32_t wt = lane < (unsigned)NW ? red.wtot[lane] : 0u;
        const uint32_t before = __reduce_add_sync(0xFFFFFFFFu, lane < warp ? wt : 0u);
        const uint32_t nlist = __reduce_add_sync(0xFFFFFFFFu, wt) >> 16;
        uint32_t run = before + inc - v;
        uint32_t li = run >> 16;
        run &= 0xFFFFu;
        // the word's first place and its slots' running counts (the counters
        // are read again rather than kept in registers across the barrier)
#pragma unroll
        for (int j = 0; j < IPT / 4; ++j) {
            uint4* qp = quad(j);
            uint4 q = *qp;
            auto start = [&](uint32_t w) {
                const uint32_t m = w * 0x01010101u;  // byte k: keys in slots 0..k of the word
                const uint32_t p = (run << 18) | ((m >> 4) & 0x3F000u) | ((m >> 2) & 0xFC0u) | (m & 0x3Fu);
                run += m >> 24;
                return p;
            };
            q.x = start(q.x);
            q.y = start(q.y);
            q.z = start(q.z);
            q.w = start(q.w);
            *qp = q;
        }
        __syncthreads();
        // 4. deal the keys into their places, and list the slots of several
#pragma unroll
        for (int r = 0; r < IPT; ++r) {
            if (r < own) {
                const uint32_t w = *reinterpret_cast<const uint32_t*>(ctr + (pr[r] & 0xFFFCu));
                const uint32_t rank = pr[r] >> 16;
                s[(w >> 18) + (((w << 6) >> ((pr[r] & 3u) * 6u)) & 63u) + rank] = key[r];
                if (rank == 1u) list[li++] = (uint16_t)pr[r];
            }
        }
        refill();
        __syncthreads();
        // 5. the keys of a slot of several are in dealing order: one thread
        // puts them in key order, in place
        for (uint32_t q = tid; q < nlist; q += THREADS) {
            const uint32_t e = list[q];
            const uint32_t pa = e & 0xFFFCu, k = e & 3u;
            const uint32_t w = *reinterpret_cast<const uint32_t*>(ctr + pa);
            const uint32_t na = ctr_swizzle<IPT>(pa) + 4u;  // the next word's logical offset
            const uint32_t wn =
                na < S * 4 ? *reinterpret_cast<const uint32_t*>(ctr + ctr_swizzle<IPT>(na)) : c << 18;
            const uint32_t w6 = w << 6;
            const uint32_t f0 = (w6 >> (k * 6u)) & 63u;
            const uint32_t f1 =  // (places are 14 bits: the difference is taken modulo 2^14)
                k == 3u ? ((wn >> 18) - (w >> 18)) & 0x3FFFu : (w6 >> (k * 6u + 6u)) & 63u;
            const uint32_t a0 = (w >> 18) + f0, n = f1 - f0;
            if (n == 2) {
                const K x0 = s[a0], x1 = s[a0 + 1];
                if (x1 < x0) {
                    s[a0] = x1;
                    s[a0 + 1] = x0;
                }
            } else {
                for (uint32_t i = a0 + 1; i < a0 + n; ++i) {
                    const K x = s[i];
                    uint32_t t = i;
                    for (; t > a0; --t) {
                        const K y = s[t - 1];
                        if (!(x < y)) break;
                        s[t] = y;
                    }
                    s[t] = x;
                }
            }
        }
        __syncthreads();
        // 6. every key is in its final place
        if constexpr (sizeof(K) == 8) {
            // (unrolled in full, its registers would push out the next keys)
            for (uint32_t p = tid; p < c; p += THREADS) store(p, s[p]);
        } else {
#pragma unroll
            for (int r = 0; r < IPT; ++r)
                if (r < own) store((uint32_t)r * THREADS + tid, s[(uint32_t)r * THREADS + tid]);
        }
    } else if constexpr (MODE != SLOT_HAND) {
        // uneven spread: bitonic leaves + merge path on the same keys
#pragma unroll
        for (int r = 0; r < IPT; ++r) {
            const uint32_t i = (uint32_t)r * THREADS + tid;
            if (i < c) s[pidx(i)] = key[r];
        }
        block_merge_sort<K, THREADS, IPT>(s, c);
        for (uint32_t i = tid; i < c; i += THREADS) store(i, s[pidx(i)]);
        refill();  // (after the merge, which needs the registers)
        __syncthreads();
    } else {
        if (tid == 0) uneven();
        refill();
    }
    return even ? SLOT_EVEN : SLOT_UNEVEN;
}

}  // namespace s512
