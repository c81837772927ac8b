// Exclusive prefix sums of int32 counts into int64 offsets, the total at [n]:
// photon rows per frame, candidates per frame and per likelihood row, phaser
// rows per (rotation, detector pixel).
//
// A tile is SCAN_TILE counts, scanned by one CTA with coalesced reads and
// warp shuffles.  Up to SCAN_ONE tiles one CTA walks them in order (one
// launch).  Above that three launches spread over the GPU, with no scratch:
// a tile's own sum is parked in the first offset the tile owns, off[tile *
// SCAN_TILE], one CTA turns those into the tiles' starts, and each tile then
// reads its start before it overwrites it.  What bounds it is the 4 + 8
// bytes per count; the earlier form, one CTA whose threads each walked a
// contiguous run of n / 1024 counts (uncoalesced, one load in flight), took
// 9.69 ms for the 10.2 M counts of a 101^2 detector's pixel maps at 1,000
// rotations, this one 0.05 ms; 73 k counts took 0.05 ms, now 0.006 ms.
#include "rspi_common.cuh"

namespace {

constexpr int SCAN_THREADS = 1024;
constexpr int SCAN_PER = 4;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_PER;
constexpr int SCAN_ONE = 4;   // tiles one CTA walks: four cost what three launches do

// Exclusive prefix of v over the CTA's threads, and the CTA's total in *total.
__device__ __forceinline__ long long cta_scan(long long v, long long *warp_tot,
                                              long long *total) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    long long x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const long long y = __shfl_up_sync(RSPI_FULL_MASK, x, o);
        if (lane >= o) x += y;
    }
    __syncthreads();   // the previous call's readers are done
    if (lane == 31) warp_tot[wid] = x;
    __syncthreads();
    long long w = warp_tot[lane];   // 32 warps
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const long long y = __shfl_up_sync(RSPI_FULL_MASK, w, o);
        if (lane >= o) w += y;
    }
    const long long before = __shfl_sync(RSPI_FULL_MASK, w, wid > 0 ? wid - 1 : 0);
    *total = __shfl_sync(RSPI_FULL_MASK, w, 31);
    return (wid > 0 ? before : 0) + x - v;
}

// One tile from `carry` on: its offsets written, its total returned.
__device__ __forceinline__ long long scan_tile(const int *__restrict__ cnt, long long n,
                                               long long tile, long long carry,
                                               long long *__restrict__ off,
                                               long long *warp_tot) {
    const long long i0 = tile * SCAN_TILE + (long long)threadIdx.x * SCAN_PER;
    int c[SCAN_PER];
    long long sum = 0;
#pragma unroll
    for (int k = 0; k < SCAN_PER; ++k) {
        c[k] = i0 + k < n ? cnt[i0 + k] : 0;
        sum += c[k];
    }
    long long total;
    long long at = carry + cta_scan(sum, warp_tot, &total);
#pragma unroll
    for (int k = 0; k < SCAN_PER; ++k) {
        if (i0 + k < n) off[i0 + k] = at;
        at += c[k];
    }
    return total;
}

__global__ void __launch_bounds__(SCAN_THREADS)
k_scan_one(const int *__restrict__ cnt, long long n, long long *__restrict__ off) {
    __shared__ long long warp_tot[32];
    const long long tiles = (n + SCAN_TILE - 1) / SCAN_TILE;
    long long carry = 0;
    for (long long t = 0; t < tiles; ++t) carry += scan_tile(cnt, n, t, carry, off, warp_tot);
    if (threadIdx.x == 0) off[n] = carry;
}

// off[tile * SCAN_TILE] = the tile's sum
__global__ void __launch_bounds__(SCAN_THREADS)
k_scan_sums(const int *__restrict__ cnt, long long n, long long *__restrict__ off) {
    __shared__ long long warp_tot[32];
    const long long i0 = (long long)blockIdx.x * SCAN_TILE;
    long long sum = 0;
#pragma unroll
    for (int k = 0; k < SCAN_PER; ++k) {
        const long long i = i0 + (long long)k * SCAN_THREADS + threadIdx.x;
        sum += i < n ? cnt[i] : 0;
    }
    long long total;
    cta_scan(sum, warp_tot, &total);
    if (threadIdx.x == 0) off[i0] = total;
}

// The parked tile sums to tile starts (one CTA), the total to off[n].
__global__ void __launch_bounds__(SCAN_THREADS)
k_scan_starts(long long n, long long *__restrict__ off) {
    __shared__ long long warp_tot[32];
    const long long tiles = (n + SCAN_TILE - 1) / SCAN_TILE;
    long long carry = 0;
    for (long long t0 = 0; t0 < tiles; t0 += SCAN_THREADS) {
        const long long t = t0 + threadIdx.x;
        const long long v = t < tiles ? off[t * SCAN_TILE] : 0;
        long long total;
        const long long at = carry + cta_scan(v, warp_tot, &total);
        if (t < tiles) off[t * SCAN_TILE] = at;
        carry += total;
    }
    if (threadIdx.x == 0) off[n] = carry;
}

__global__ void __launch_bounds__(SCAN_THREADS)
k_scan_tiles(const int *__restrict__ cnt, long long n, long long *off) {
    __shared__ long long warp_tot[32];
    const long long carry = off[(long long)blockIdx.x * SCAN_TILE];
    __syncthreads();   // every thread has the start before thread 0 overwrites it
    scan_tile(cnt, n, blockIdx.x, carry, off, warp_tot);
}

}  // namespace

int rspi_scan_i32(const int *cnt, long long n, long long *off, cudaStream_t stream) {
    const long long tiles = (n + SCAN_TILE - 1) / SCAN_TILE;
    if (tiles > 0x7fffffffLL) return RSPI_ERR_ARG;
    if (tiles <= SCAN_ONE) {
        k_scan_one<<<1, SCAN_THREADS, 0, stream>>>(cnt, n, off);
    } else {
        k_scan_sums<<<(unsigned)tiles, SCAN_THREADS, 0, stream>>>(cnt, n, off);
        k_scan_starts<<<1, SCAN_THREADS, 0, stream>>>(n, off);
        k_scan_tiles<<<(unsigned)tiles, SCAN_THREADS, 0, stream>>>(cnt, n, off);
    }
    RSPI_RETURN_LAUNCH();
}

extern "C" int rspi_scan_launches(long long n) {
    return (n + SCAN_TILE - 1) / SCAN_TILE <= SCAN_ONE ? 1 : 3;
}

extern "C" int rspi_scan_rows(const int *frame_rows, long long n_data, long long *row_off,
                              cudaStream_t stream) {
    if (n_data <= 0 || !frame_rows || !row_off) return RSPI_ERR_ARG;
    return rspi_scan_i32(frame_rows, n_data, row_off, stream);
}
