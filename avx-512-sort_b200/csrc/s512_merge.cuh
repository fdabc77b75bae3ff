// s512_merge.cuh -- merge-path merging of sorted runs in global memory.
//
// The reference merges sorted runs in its OpenMP drivers: SortOmpMerge and
// SortOmpMergeDeps call std::inplace_merge on neighbouring chunks level by
// level (sort512.hpp:6045, 6092); SortOmpParMerge calls
// ParallelInplace::parallelMergeInPlace (parallelInplace.hpp:210-306), which
// splits a merge between threads with FindMedian (78-135) -- a binary search
// for where a diagonal of the merge crosses the two runs -- and rotates the
// middle parts into place (reorderShifting, 31-75).
//
// On the GPU the same split is the merge path: the output of a pair of runs
// is cut into tiles of TILE outputs; corank_kernel finds, for every tile
// boundary at once, how many of the first d outputs come from the left run
// (binary search); merge_kernel then loads each tile's two input slices into
// shared memory and every thread merges its own EPT outputs after a second,
// shared-memory co-rank search.  Comparisons use the element type's own `<`
// and take from the left run on ties, which is std::inplace_merge's (stable)
// result.
//
// What bounds it: HBM for large merges.  Per output the tile costs one shared
// load and one compare (each thread keeps the heads of its two runs in
// registers), the tile's loads are all in flight at once, and the outputs are
// staged in a padded layout: a thread writes 16 consecutive outputs, which
// unpadded put all lanes of a store on one bank.  33.5M doubles: co-ranks 22
// -> 18 us, merge 271 -> 134 us; floor 82 us.
#pragma once

#include "s512_common.cuh"

namespace s512 {

// One pair of adjacent sorted runs to merge: a = src[a0, a0+la), b = src[b0, b0+lb)
// into dst[out0, out0+la+lb).  tile0 = first tile of this pair.
struct MergePair {
    uint64_t a0, la, b0, lb, out0;
    uint32_t tile0, ntiles;
};

// The pairs of one level: up to MERGE_INLINE travel with the launch, more in
// device memory.
constexpr int MERGE_INLINE = 16;
struct MergePairs {
    MergePair p[MERGE_INLINE];
    const MergePair* more;  // all pairs, when there are more than MERGE_INLINE
    uint32_t n;
    __device__ __forceinline__ MergePair of_tile(uint32_t t) const {
        const MergePair* q = n > MERGE_INLINE ? more : p;
        uint32_t lo = 0, hi = n;
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (q[mid].tile0 <= t) lo = mid; else hi = mid;
        }
        return q[lo];
    }
};

constexpr int MERGE_THREADS = 256;
constexpr int MERGE_EPT = 16;
constexpr int MERGE_TILE = MERGE_THREADS * MERGE_EPT;  // 4096 outputs per tile
__device__ __forceinline__ uint32_t merge_pad(uint32_t e) { return e + (e >> 4); }  // place of staged output e

// smallest i in [max(0,d-lb), min(d,la)] such that a[i] > b[d-1-i] (ties -> a first)
template <typename I, typename AF, typename BF>
__device__ __forceinline__ I corank(I d, I la, I lb, AF a, BF b) {
    I lo = d > lb ? d - lb : 0;
    I hi = d < la ? d : la;
    while (lo < hi) {
        const I mid = (lo + hi) >> 1;
        if (b(d - 1 - mid) < a(mid)) hi = mid;
        else lo = mid + 1;
    }
    return lo;
}

// co-rank of every tile start; corank_out[t] = number of left-run keys among
// the pair's first (t - tile0) * TILE outputs.  CR_LANES lanes per tile probe
// at once and narrow the range CR_LANES + 1 fold for one round trip to memory
// (a thread per tile: 25 round trips, 22 us for 8192 tiles of 33.5M doubles; a
// warp per tile: 5, but 2.6M scattered reads, 31 us; 8 lanes: 18 us).
constexpr int CR_LANES = 8;
template <typename T>
__global__ void __launch_bounds__(256) corank_kernel(const T* __restrict__ src, MergePairs pairs, uint32_t ntiles,
                                                     uint64_t* __restrict__ corank_out) {
    const uint32_t t = blockIdx.x * (256 / CR_LANES) + threadIdx.x / CR_LANES;
    const unsigned lane = threadIdx.x & 31u, g = lane % CR_LANES;
    const T *a = src, *b = src;
    uint64_t d = 0, lo = 0, hi = 0;
    if (t < ntiles) {
        const MergePair p = pairs.of_tile(t);
        d = (uint64_t)(t - p.tile0) * MERGE_TILE;
        a += p.a0;
        b += p.b0;
        lo = d > p.lb ? d - p.lb : 0;
        hi = d < p.la ? d : p.la;
    }
    while (__any_sync(0xFFFFFFFFu, lo < hi)) {  // the answer is in [lo, hi]; past(i) is false, then true
        const uint64_t step = (hi - lo + CR_LANES) / (CR_LANES + 1);
        const uint64_t i = lo + (g + 1) * step - 1;  // probes lo + step - 1, lo + 2 step - 1, ...
        const bool past = lo >= hi || i >= hi || b[d - 1 - i] < a[i];
        const unsigned m = (__ballot_sync(0xFFFFFFFFu, past) >> (lane - g)) & ((1u << CR_LANES) - 1u);
        if (lo < hi) {
            const uint32_t first = m ? (uint32_t)__ffs(m) - 1 : (uint32_t)CR_LANES;  // probes before it are not past
            lo += first * step;
            if (first < (uint32_t)CR_LANES) hi = min(hi, lo + step - 1);
            lo = min(lo, hi);
        }
    }
    if (t < ntiles && g == 0) corank_out[t] = lo;
}

template <typename T>
__global__ void __launch_bounds__(MERGE_THREADS) merge_kernel(const T* __restrict__ src, T* __restrict__ dst,
                                                              MergePairs pairs, uint32_t ntiles,
                                                              const uint64_t* __restrict__ coranks) {
    // one tile's two input slices, left then right (na + nb <= MERGE_TILE);
    // each thread merges its outputs into registers, then writes them back
    // here for a coalesced store
    __shared__ T buf[MERGE_TILE + MERGE_TILE / 16 + 1];
    for (uint32_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const MergePair p = pairs.of_tile(t);
        const uint64_t total = p.la + p.lb;
        const uint64_t d0 = (uint64_t)(t - p.tile0) * MERGE_TILE;
        const uint64_t d1 = d0 + MERGE_TILE < total ? d0 + MERGE_TILE : total;
        const uint64_t i0 = coranks[t];
        const uint64_t i1 = (t + 1 < p.tile0 + p.ntiles) ? coranks[t + 1] : p.la;
        const uint32_t na = (uint32_t)(i1 - i0), nout = (uint32_t)(d1 - d0);
        // element k of the tile's input: the left slice, then the right one
        const T* sa = src + p.a0 + i0;
        const T* sb = src + p.b0 + (d0 - i0) - na;
        T out[MERGE_EPT];
#pragma unroll
        for (int r = 0; r < MERGE_EPT; ++r) {
            const uint32_t k = r * MERGE_THREADS + threadIdx.x;
            if (k < nout) out[r] = (k < na ? sa : sb)[k];
        }
#pragma unroll
        for (int r = 0; r < MERGE_EPT; ++r) {
            const uint32_t k = r * MERGE_THREADS + threadIdx.x;
            if (k < nout) buf[k] = out[r];
        }
        __syncthreads();
        const uint32_t o0 = threadIdx.x * MERGE_EPT;
        uint32_t cnt = 0;
        if (o0 < nout) {
            uint32_t ia = corank<uint32_t>(o0, na, nout - na, [&](uint32_t i) { return buf[i]; },
                                           [&](uint32_t j) { return buf[na + j]; });
            uint32_t ib = na + o0 - ia;
            cnt = nout - o0 < (uint32_t)MERGE_EPT ? nout - o0 : (uint32_t)MERGE_EPT;
            T va = buf[ia], vb = buf[ib];  // (past a slice's end: another key of the buffer, not used)
#pragma unroll
            for (int k = 0; k < MERGE_EPT; ++k) {
                const bool take_a = ib >= nout || (ia < na && !(vb < va));
                out[k] = take_a ? va : vb;
                const uint32_t next = (take_a ? ia : ib) + 1;
                const T v = buf[next < (uint32_t)MERGE_TILE ? next : (uint32_t)MERGE_TILE];
                if (take_a) {
                    ia = next;
                    va = v;
                } else {
                    ib = next;
                    vb = v;
                }
            }
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < MERGE_EPT; ++k)
            if ((uint32_t)k < cnt) buf[merge_pad(o0 + k)] = out[k];
        __syncthreads();
#pragma unroll
        for (int r = 0; r < MERGE_EPT; ++r) {
            const uint32_t k = r * MERGE_THREADS + threadIdx.x;
            if (k < nout) dst[p.out0 + d0 + k] = buf[merge_pad(k)];
        }
        __syncthreads();
    }
}

}  // namespace s512
