// s512_partition2.cuh -- the two-way partition behind Partition512.
//
// Partition512 (sort512.hpp:5729-5819 int, 5821-5912 double; kv
// sort512kv.hpp:5959-6082) moves every element <= pivot before every element
// > pivot inside [left, right] and returns the first index of the > side.  The
// reference walks the range from both ends with compress-stores.  Here every
// warp owns a run of consecutive elements.  A first launch counts each run's
// lows while it copies the range to scratch; a second one adds up the counts
// before each run and writes lows forward from the start and highs backward
// from the end of the caller's range.  The comparison is the reference's own:
// `x <= pivot` on the caller's type (so a NaN double goes to the high side, as
// with _CMP_LE_OQ).
//
// Bound by HBM: two reads and two writes of the range, the least for a result
// in place.  Warps need no barrier and no other warp: a single pass with a
// decoupled look-back has the same traffic (its result is copied back), but
// its tiles start only as fast as the look-back reaches an inclusive count.
// 20M doubles (160 MB): 201 + 56 us with the look-back and the copy, 155 + 55
// with a look-back of 256 tiles a step, 53 + 58 us here; the floor is 98 us.
#pragma once

#include "s512_common.cuh"

namespace s512 {

constexpr int P2_THREADS = 256;
constexpr int P2_WARPS = P2_THREADS / 32;
constexpr int P2_ROWS = 8;                    // rows of 32 elements a warp has in flight
constexpr int P2_MIN_RUN = 32 * P2_ROWS;      // smallest run worth a warp

struct Part2Ctl {
    uint32_t err;
    uint32_t never_set;            // testing: a flag nothing writes (the injected wait)
    unsigned long long total_low;
};

// How a range of n elements is split: `blocks` blocks, `run` elements a warp.
struct Part2Shape {
    uint32_t blocks;
    uint64_t run;
};
__host__ inline Part2Shape part2_shape(uint64_t n, uint32_t max_blocks) {
    const uint64_t want = (n + (uint64_t)P2_MIN_RUN * P2_WARPS - 1) / ((uint64_t)P2_MIN_RUN * P2_WARPS);
    Part2Shape s;
    s.blocks = want < max_blocks ? (want ? (uint32_t)want : 1u) : max_blocks;
    const uint64_t warps = (uint64_t)s.blocks * P2_WARPS;
    s.run = ((n + warps - 1) / warps + 31) / 32 * 32;
    return s;
}

// Bytes of the counts: a word per block, then one per warp.
__host__ __device__ constexpr size_t part2_count_words(size_t blocks) { return blocks * (1 + P2_WARPS); }

// Launch 1: the range copied to scratch, and the lows of every run (counts:
// per block, then per warp).  Runs are walked from the back, so that what the
// second launch reads first was written last and is still in L2.
template <typename T, bool KV>
__global__ void __launch_bounds__(P2_THREADS)
    part2_count_kernel(const T* __restrict__ in, const int* __restrict__ vin, T* __restrict__ tmp,
                       int* __restrict__ vtmp, uint64_t n, T pivot, uint64_t run,
                       unsigned long long* __restrict__ counts, Part2Ctl* ctl, int inject_timeout) {
    __shared__ unsigned long long total;
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) total = 0;
    __syncthreads();
    const uint64_t gw = (uint64_t)blockIdx.x * P2_WARPS + warp;
    const uint64_t first = min(gw * run, n), end = min(first + run, n);
    unsigned long long low = 0;
    for (uint64_t step = (end - first + P2_MIN_RUN - 1) / P2_MIN_RUN; step-- > 0;) {
        const uint64_t base = first + step * P2_MIN_RUN + lane;
        T x[P2_ROWS];
        int v[P2_ROWS];
#pragma unroll
        for (int r = 0; r < P2_ROWS; ++r) {
            const uint64_t i = base + r * 32;
            x[r] = pivot;
            v[r] = 0;
            if (i < end) {
                x[r] = in[i];
                if (KV) v[r] = vin[i];
            }
        }
#pragma unroll
        for (int r = 0; r < P2_ROWS; ++r) {
            const uint64_t i = base + r * 32;
            if (i < end) {
                low += x[r] <= pivot ? 1u : 0u;
                tmp[i] = x[r];
                if (KV) vtmp[i] = v[r];
            }
        }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) low += __shfl_xor_sync(0xFFFFFFFFu, low, d);
    if (lane == 0) {
        counts[gridDim.x + gw] = low;
        atomicAdd(&total, low);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        counts[blockIdx.x] = total;
        if (blockIdx.x == 0) {
            uint32_t err = DEV_ERR_NONE;
            if (inject_timeout) {
                // injected failure: a wait on a flag that nothing sets, with a
                // short bound; the second launch then writes nothing
                uint32_t spins = 0;
                while (*(volatile uint32_t*)&ctl->never_set != 0xA5A5A5A5u && ++spins < 1024u) __nanosleep(100);
                err = DEV_ERR_TIMEOUT;
            }
            ctl->err = err;
        }
    }
}

// Launch 2 (the same blocks): every element to its place.
template <typename T, bool KV>
__global__ void __launch_bounds__(P2_THREADS)
    part2_scatter_kernel(const T* __restrict__ tmp, const int* __restrict__ vtmp, T* __restrict__ out,
                         int* __restrict__ vout, uint64_t n, T pivot, uint64_t run,
                         const unsigned long long* __restrict__ counts, Part2Ctl* ctl) {
    __shared__ unsigned long long part[P2_WARPS];
    if (ctl->err) return;
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    // lows of the earlier blocks, then of this block's earlier warps
    unsigned long long s = 0;
    for (uint32_t b = threadIdx.x; b < blockIdx.x; b += P2_THREADS) s += counts[b];
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, d);
    if (lane == 0) part[warp] = s;
    __syncthreads();
    const uint64_t gw = (uint64_t)blockIdx.x * P2_WARPS + warp;
    uint64_t lows = 0;  // lows before the row
#pragma unroll
    for (int w = 0; w < P2_WARPS; ++w) {
        lows += part[w];
        if (w < (int)warp) lows += counts[gridDim.x + (uint64_t)blockIdx.x * P2_WARPS + w];
    }
    if (blockIdx.x == gridDim.x - 1 && warp == P2_WARPS - 1 && lane == 0)
        ctl->total_low = lows + counts[gridDim.x + gw];
    const uint64_t first = min(gw * run, n), end = min(first + run, n);
    for (uint64_t at = first; at < end; at += P2_MIN_RUN) {
        const uint64_t base = at + lane;
        T x[P2_ROWS];
        int v[P2_ROWS];
#pragma unroll
        for (int r = 0; r < P2_ROWS; ++r) {
            const uint64_t i = base + r * 32;
            x[r] = pivot;
            v[r] = 0;
            if (i < end) {
                x[r] = tmp[i];
                if (KV) v[r] = vtmp[i];
            }
        }
#pragma unroll
        for (int r = 0; r < P2_ROWS; ++r) {
            const uint64_t i = base + r * 32;
            const bool low = i < end && x[r] <= pivot;
            const unsigned m = __ballot_sync(0xFFFFFFFFu, low);
            const uint64_t before = lows + __popc(m & lt);
            const uint64_t o = low ? before : n - 1 - (i - before);
            if (i < end) {
                out[o] = x[r];
                if (KV) vout[o] = v[r];
            }
            lows += __popc(m);
        }
    }
}

// Both launches.  counts: part2_count_words(shape.blocks) words.
template <typename T, bool KV>
static cudaError_t launch_part2(T* data, int* values, T* tmp, int* vtmp, uint64_t n, T pivot, Part2Shape sh,
                                unsigned long long* counts, Part2Ctl* ctl, int inject_timeout, cudaStream_t st) {
    part2_count_kernel<T, KV><<<sh.blocks, P2_THREADS, 0, st>>>(data, values, tmp, vtmp, n, pivot, sh.run, counts, ctl,
                                                                inject_timeout);
    part2_scatter_kernel<T, KV><<<sh.blocks, P2_THREADS, 0, st>>>(tmp, vtmp, data, values, n, pivot, sh.run, counts,
                                                                  ctl);
    return cudaGetLastError();
}

}  // namespace s512
