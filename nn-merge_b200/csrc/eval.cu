// Recall of a k-NN graph on the device (the reference's Evaluator,
// evaluator.cpp:258-295, with the ground truth computed here instead of read
// from a file).
//
// For each evaluated row r: t_r = the atop-th smallest distance from r to
// every other row (exact brute force, the reference's sequential FP32 sum);
// a hit is one of the graph's first atop ids of r whose distance is <= t_r.
// recall = hits / (rows x atop).  Where no two rows tie at the atop-th
// distance this is the size of the intersection of the graph's first atop
// ids with the exact atop nearest ids (getKGraphRecall); tied rows count as
// hits either way.
//
// k_kth: 8 warps per block, EQ evaluated rows per warp; the block streams its
// share of the data set through shared memory in tiles of 64 rows; lane l
// measures tile rows l and l + 32 against the warp's EQ rows (EQ x 2
// distances at a time: 10 shared-memory wavefronts for 48 FP32 instructions
// per four components, where one row and one tile row at a time took 5 for
// 12 and was bound by the reads) and keeps the 16 smallest of each in
// registers; the warp then merges the 32 lists to its share's atop smallest.
// The data set is split over blockIdx.y so that a few hundred evaluated rows
// still fill the SMs; k_hits takes the atop-th smallest of the shares.
// 1,000 rows against 100,000 x 128: 2.1 ms, against 7.75 ms for one row a warp
// in one pass of 125 blocks.
#include <algorithm>
#include <cmath>
#include <vector>

#include "nnm_common.cuh"
#include "nnm_eval.h"
#include "nnm_launch.h"

namespace nnm {
namespace {
constexpr unsigned FULL = 0xffffffffu;
constexpr uint32_t EW = 8;   // warps per block
constexpr uint32_t EQ = 2;   // evaluated rows per warp
constexpr uint32_t EB = EW * EQ;
constexpr uint32_t ET = 64;  // data rows per shared-memory tile
constexpr uint32_t MAX_SPLIT = 32;
constexpr int EA = EVAL_MAX_ATOP;

// part[(row * splits + split) * EA + t]: the t-th smallest distance (t < atop)
// from evaluated row `row` to the other rows of the split's tiles.
template <int M>
__global__ void __launch_bounds__(EW * 32) k_kth(const float* __restrict__ x, uint32_t n, uint32_t dp,
                                                 const uint32_t* __restrict__ rows, uint32_t nrows, uint32_t atop,
                                                 uint32_t tiles_per, float* __restrict__ part) {
    extern __shared__ __align__(16) float sm[];
    const uint32_t st = dp + 4;  // row stride: a quarter-warp's float4 reads fall in distinct banks
    float* tile = sm;
    float* qs = sm + ET * st;
    const uint32_t w = threadIdx.x >> 5, lane = threadIdx.x & 31, r0 = blockIdx.x * EB, dq = dp / 4;
    for (uint32_t i = threadIdx.x; i < EB * dp; i += blockDim.x) {
        const uint32_t e = i / dp, c = i - e * dp;
        qs[e * st + c] = r0 + e < nrows ? x[(size_t)rows[r0 + e] * dp + c] : 0.f;
    }
    uint32_t self[EQ];
    float best[EQ][EA];
#pragma unroll
    for (uint32_t e = 0; e < EQ; e++) {
        self[e] = r0 + w * EQ + e < nrows ? rows[r0 + w * EQ + e] : 0xffffffffu;
#pragma unroll
        for (int q = 0; q < EA; q++) best[e][q] = INFINITY;
    }
    const bool active = r0 + w * EQ < nrows;
    const uint32_t t_end = min((n + ET - 1) / ET, (blockIdx.y + 1) * tiles_per);
    for (uint32_t t = blockIdx.y * tiles_per; t < t_end; t++) {
        const uint32_t t0 = t * ET, nt = min(ET, n - t0);
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < nt * dq; i += blockDim.x) {
            const uint32_t rr = i / dq, c4 = i - rr * dq;
            *reinterpret_cast<float4*>(tile + rr * st + 4 * c4) =
                *reinterpret_cast<const float4*>(x + (size_t)(t0 + rr) * dp + 4 * c4);
        }
        __syncthreads();
        if (!active) continue;
        float acc[EQ][2];
#pragma unroll
        for (uint32_t e = 0; e < EQ; e++) acc[e][0] = acc[e][1] = 0.f;
        const float4* b0 = reinterpret_cast<const float4*>(tile + lane * st);
        const float4* b1 = reinterpret_cast<const float4*>(tile + (lane + 32) * st);
        const float4* qr = reinterpret_cast<const float4*>(qs + w * EQ * st);
#pragma unroll 2
        for (uint32_t c = 0; c < dq; c++) {
            const float4 v0 = b0[c], v1 = b1[c];
#pragma unroll
            for (uint32_t e = 0; e < EQ; e++) {
                const float4 q = qr[e * (st / 4) + c];
                acc[e][0] = dist_step<M>(acc[e][0], q.x, v0.x);
                acc[e][1] = dist_step<M>(acc[e][1], q.x, v1.x);
                acc[e][0] = dist_step<M>(acc[e][0], q.y, v0.y);
                acc[e][1] = dist_step<M>(acc[e][1], q.y, v1.y);
                acc[e][0] = dist_step<M>(acc[e][0], q.z, v0.z);
                acc[e][1] = dist_step<M>(acc[e][1], q.z, v1.z);
                acc[e][0] = dist_step<M>(acc[e][0], q.w, v0.w);
                acc[e][1] = dist_step<M>(acc[e][1], q.w, v1.w);
            }
        }
#pragma unroll
        for (uint32_t e = 0; e < EQ; e++)
#pragma unroll
            for (uint32_t h = 0; h < 2; h++) {
                const uint32_t j = lane + 32 * h;
                const float d = acc[e][h];
                if (j < nt && t0 + j != self[e] && d < best[e][EA - 1]) {
                    best[e][EA - 1] = d;
#pragma unroll
                    for (int q = EA - 1; q > 0; q--)
                        if (best[e][q] < best[e][q - 1]) {
                            const float tv = best[e][q];
                            best[e][q] = best[e][q - 1];
                            best[e][q - 1] = tv;
                        }
                }
            }
    }
    // the atop smallest of the 32 sorted lists: rounds of taking the smallest
    // list head
#pragma unroll
    for (uint32_t e = 0; e < EQ; e++) {
        const uint32_t row = r0 + w * EQ + e;
        if (row >= nrows) break;
        float* out = part + ((size_t)row * gridDim.y + blockIdx.y) * EA;
        for (uint32_t t = 0; t < atop; t++) {
            float m = best[e][0];
            uint32_t ml = lane;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const float om = __shfl_xor_sync(FULL, m, o);
                const uint32_t ol = __shfl_xor_sync(FULL, ml, o);
                if (om < m || (om == m && ol < ml)) {
                    m = om;
                    ml = ol;
                }
            }
            if (lane == 0) out[t] = m;
            if (lane == ml) {
#pragma unroll
                for (int q = 0; q < EA - 1; q++) best[e][q] = best[e][q + 1];
                best[e][EA - 1] = INFINITY;
            }
        }
    }
}

// Warp per evaluated row: the atop-th smallest of its shares' lists (lane l
// walks share l's), then the hits among the graph's first atop ids.  ids:
// row i of the graph at ids + i k, or (by_eval) the w-th evaluated row's.
__global__ void k_hits(const float* __restrict__ x, uint32_t dp, int metric, const uint32_t* __restrict__ ids,
                       uint32_t k, bool by_eval, const uint32_t* __restrict__ rows, uint32_t nrows, uint32_t atop,
                       uint32_t n, const float* __restrict__ part, uint32_t splits,
                       unsigned long long* __restrict__ hits) {
    const uint32_t w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (w >= nrows) return;
    const float* mine = part + ((size_t)w * splits + lane) * EA;
    uint32_t at = 0;
    float head = lane < splits ? mine[0] : INFINITY, kth = INFINITY;
    for (uint32_t t = 0; t < atop; t++) {
        float m = head;
        uint32_t ml = lane;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float om = __shfl_xor_sync(FULL, m, o);
            const uint32_t ol = __shfl_xor_sync(FULL, ml, o);
            if (om < m || (om == m && ol < ml)) {
                m = om;
                ml = ol;
            }
        }
        kth = m;
        if (lane == ml) head = ++at < atop && lane < splits ? mine[at] : INFINITY;
    }
    const uint32_t row = rows[w];
    bool hit = false;
    if (lane < atop) {
        const uint32_t id = ids[(size_t)(by_eval ? w : row) * k + lane] & ID_MASK;
        if (id < n && id != row)
            hit = dist_seq_rt(metric, x + (size_t)row * dp, x + (size_t)id * dp, (int)dp) <= kth;
    }
    const uint32_t c = __popc(__ballot_sync(FULL, hit));
    if (lane == 0 && c) atomicAdd(hits, (unsigned long long)c);
}
}  // namespace

int graph_recall_dev(Ctx& ctx, const float* x, uint32_t n, uint32_t dp, int metric, const uint32_t* ids, uint32_t k,
                     bool by_eval, const uint32_t* rows, uint32_t nrows, uint32_t atop, double* recall) {
    if (!nrows) {
        *recall = 0.0;
        return 0;
    }
    const auto kth = metric == L2 ? k_kth<L2> : metric == L1 ? k_kth<L1> : k_kth<CHI2>;
    const size_t smem = ((size_t)ET + EB) * (dp + 4) * 4;
    int nsm = 148, per_sm = 1;
    NNM_CUDA_TRY(cudaFuncSetAttribute(kth, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    NNM_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, ctx.device));
    NNM_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kth, EW * 32, smem));
    // shares of the data set: up to a wave of blocks, at least 8 tiles each
    const uint32_t row_blocks = (nrows + EB - 1) / EB, tiles = (n + ET - 1) / ET;
    const uint32_t wave = (uint32_t)nsm * (uint32_t)std::max(per_sm, 1);
    uint32_t splits = std::max(1u, std::min({wave / row_blocks, tiles / 8, MAX_SPLIT}));
    const uint32_t tiles_per = (tiles + splits - 1) / splits;
    splits = (tiles + tiles_per - 1) / tiles_per;
    DevBuf& buf = ctx.ws.misc;
    NNM_CUDA_TRY(buf.ensure(64 + (size_t)nrows * splits * EA * 4));
    unsigned long long* hits = buf.as<unsigned long long>();
    float* part = reinterpret_cast<float*>(buf.as<unsigned char>() + 64);
    cudaStream_t st = ctx.stream;
    NNM_CUDA_TRY(cudaMemsetAsync(hits, 0, 8, st));
    kth<<<dim3(row_blocks, splits), EW * 32, smem, st>>>(x, n, dp, rows, nrows, atop, tiles_per, part);
    k_hits<<<(nrows + 7) / 8, 256, 0, st>>>(x, dp, metric, ids, k, by_eval, rows, nrows, atop, n, part, splits, hits);
    count_launch(2);
    unsigned long long h = 0;
    NNM_CUDA_TRY(cudaGetLastError());
    NNM_CUDA_TRY(cudaMemcpyAsync(&h, hits, 8, cudaMemcpyDeviceToHost, st));
    NNM_CUDA_TRY(cudaStreamSynchronize(st));
    *recall = (double)h / ((double)nrows * (double)atop);
    return 0;
}

}  // namespace nnm
