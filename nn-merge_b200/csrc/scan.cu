// Device-wide exclusive prefix sums (u32 counts -> u64 offsets), used to lay
// out per-row and per-target segments (reverse lists, proposal buckets,
// random-draw ranges).  Two passes: per-tile totals, then per-tile scans whose
// blocks each add up the totals before their tile; a single tile (n <= 4096)
// needs only the second.  Up to three scans of the same length share the
// launches.  HBM-bound at large n (4 B read + 8 B written per element),
// launch-bound at small: a separate scan of the totals, one array at a time,
// was 15 launches of an exact-tier iteration and 183 of the 1,110 us the GPU
// was busy in a 2,000-row build.
#include <cstdint>
#include <cuda_runtime.h>

#include "nnm_scan.h"
#include "nnm_launch.h"

namespace nnm {
namespace {
constexpr int SCAN_THREADS = 512;
constexpr int SCAN_ITEMS = 8;
constexpr int TILE = SCAN_THREADS * SCAN_ITEMS;

__device__ __forceinline__ uint64_t block_exclusive_scan(uint64_t v, uint64_t* sh, uint64_t* total) {
    int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint64_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint64_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sh[wid] = x;
    __syncthreads();
    if (wid == 0) {
        uint64_t s = lane < (int)(blockDim.x >> 5) ? sh[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint64_t y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += y;
        }
        sh[lane] = s;
    }
    __syncthreads();
    uint64_t before = wid ? sh[wid - 1] : 0;
    if (total) *total = sh[(blockDim.x >> 5) - 1];
    __syncthreads();
    return before + x - v;
}

__device__ __forceinline__ uint32_t scan_input(const ScanJob& j, size_t i) {
    const uint32_t v = j.in[i];
    if (!j.in2) return v;
    const uint32_t w = j.in2[i];  // draws of two shuffles
    return (v ? v - 1 : 0u) + (w ? w - 1 : 0u);
}

// sums: per job, one total per tile.
__global__ void __launch_bounds__(SCAN_THREADS) k_tile_sums(ScanJobs jobs, size_t n, uint64_t* __restrict__ sums) {
    __shared__ uint64_t sh[32];
    const ScanJob& j = jobs.j[blockIdx.y];
    const size_t base = (size_t)blockIdx.x * TILE;
    uint64_t s = 0;
#pragma unroll
    for (int i = 0; i < SCAN_ITEMS; i++) {
        const size_t t = base + (size_t)i * SCAN_THREADS + threadIdx.x;
        if (t < n) s += scan_input(j, t);
    }
    uint64_t tot;
    block_exclusive_scan(s, sh, &tot);
    if (threadIdx.x == 0) sums[(size_t)blockIdx.y * gridDim.x + blockIdx.x] = tot;
}

__global__ void __launch_bounds__(SCAN_THREADS) k_tile_scan(ScanJobs jobs, size_t n,
                                                            const uint64_t* __restrict__ sums) {
    __shared__ uint64_t sh[32];
    const ScanJob& j = jobs.j[blockIdx.y];
    uint64_t before = 0;
    if (blockIdx.x) {  // the totals of the tiles before this one
        const uint64_t* js = sums + (size_t)blockIdx.y * gridDim.x;
        uint64_t p = 0;
        for (uint32_t i = threadIdx.x; i < blockIdx.x; i += SCAN_THREADS) p += js[i];
        block_exclusive_scan(p, sh, &before);
    }
    const size_t base = (size_t)blockIdx.x * TILE + (size_t)threadIdx.x * SCAN_ITEMS;
    uint32_t v[SCAN_ITEMS];
    uint64_t s = 0;
#pragma unroll
    for (int i = 0; i < SCAN_ITEMS; i++) {
        v[i] = base + i < n ? scan_input(j, base + i) : 0;
        s += v[i];
    }
    uint64_t ex = block_exclusive_scan(s, sh, nullptr) + before;
#pragma unroll
    for (int i = 0; i < SCAN_ITEMS; i++) {
        if (base + i < n) j.out[base + i] = ex;
        ex += v[i];
    }
    if (base < n && base + SCAN_ITEMS >= n) {  // thread owning the last element
        j.out[n] = ex;
        if (j.total) *j.total = ex;
        if (j.over && ex > j.cap) atomicOr(j.over, j.bit);
    }
}
}  // namespace

size_t scan_temp_elems(size_t n) { return ScanJobs::MAX * ((n + TILE - 1) / TILE) + 1; }

cudaError_t exclusive_scans(const ScanJobs& jobs, int count, size_t n, uint64_t* temp, cudaStream_t st) {
    if (n == 0) {
        for (int i = 0; i < count; i++) {
            cudaError_t e = cudaMemsetAsync(jobs.j[i].out, 0, sizeof(uint64_t), st);
            if (e == cudaSuccess && jobs.j[i].total) e = cudaMemsetAsync(jobs.j[i].total, 0, sizeof(uint64_t), st);
            if (e != cudaSuccess) return e;
        }
        return cudaSuccess;
    }
    const dim3 grid((unsigned)((n + TILE - 1) / TILE), (unsigned)count);
    if (grid.x > 1) { k_tile_sums<<<grid, SCAN_THREADS, 0, st>>>(jobs, n, temp); count_launch(); }
    k_tile_scan<<<grid, SCAN_THREADS, 0, st>>>(jobs, n, temp); count_launch();
    return cudaGetLastError();
}

cudaError_t exclusive_scan(const uint32_t* in, uint64_t* out, size_t n, uint64_t* temp, cudaStream_t st) {
    ScanJobs jobs{};
    jobs.j[0] = ScanJob{in, nullptr, out, nullptr, nullptr, 0, 0};
    return exclusive_scans(jobs, 1, n, temp, st);
}

}  // namespace nnm
