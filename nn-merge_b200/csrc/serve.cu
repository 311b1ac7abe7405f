// Fast batched LySearch (NNM_SERVE_FAST): the per-query steps of
// LySearch::knnSearch (lysearch.cpp:363-437) and nndHNSWSrch (:236-322),
// laid out for throughput rather than for the reference's float rounding.
//
// One warp per query; persistent warps pull queries from a counter, so
// queries of different beam widths balance.  (A batch whose queries all have
// a resident block takes a block per query: k_serve_team.)
//   - distances: a whole warp per distance, lane l holding components
//     [4l, 4l+4) (+128 per further float4) of the query in registers; a
//     row is one coalesced 512-byte read for d = 128.  Up to 32 distances
//     are evaluated together and reduced by a transposing butterfly (31
//     shuffles for 32 sums), after which lane j holds distance j.  The
//     summation order differs from the reference's sequential sum.
//   - greedy descent on the upper layers: the reference's rule (move to the
//     first strictly nearer neighbour of the minimum distance in list order,
//     repeat until no move) evaluated a list chunk at a time.
//   - beam: the reference keeps a result max-heap of size topk and a
//     candidate heap, and stops when the nearest candidate is farther than
//     the worst result.  Every candidate that can still be expanded is in
//     the result set, so both heaps are replaced by one array of at most
//     `beam` entries in shared memory, sorted by (distance, id), with an
//     "expanded" bit per entry: expand the first unexpanded entry, merge the
//     accepted neighbours (distance below the worst entry, or the beam not
//     full) into place (only the entries after the first new one move),
//     stop when every entry is expanded.
//   - width: a step expands the first min(width, beam / 64) unexpanded
//     entries together, reading their lists as one sequence of 32-id chunks,
//     so that the dependent loads (offsets, lists, visited bits, rows) of
//     several nodes are in flight at once; width 1 is strict best-first.
//   - visited set: one bitmap per warp slot in HBM, cleared after each query
//     from the list of ids it set, or whole where the list was too short.
#include <algorithm>
#include <cmath>

#include "nnm_hier.h"
#include "nnm_launch.h"

#pragma nv_diag_suppress 177  // every object of this file (below) uses a part of it

namespace nnm {
namespace {
constexpr unsigned FULL = 0xffffffffu;
constexpr int FW = 4;                    // warps per block
// Visited ids recorded per warp slot; a query that visits more clears its
// whole bitmap (65,536 ids took 0.8 GB an index, 1.1 in the dense form).  A
// constant: lists as long as the layer or the bitmap, as an argument, cost
// k_serve 2 to 4 % (L2 and L1, 100,000 x 128, 1,500 to 8,000 queries).
constexpr uint32_t FVCAP = 16384;
constexpr uint32_t EXP_BIT = 1u << 31;   // beam entry already expanded
constexpr uint32_t IDM = 0x7fffffffu;
constexpr uint32_t FAST_MAX_DP = 512;    // 4 float4 per lane
constexpr uint32_t WARPS = 20;                          // k_serve: warps per SM
constexpr uint32_t DENSE_WARPS = 28;                    // .. of its dense form,
constexpr size_t DENSE_SCRATCH = (size_t)387 << 20;     // with at most this much of visited bitmaps and lists (259,000 rows)
constexpr uint32_t GROUP = 4;            // 32-id chunks of a step whose loads and atomics overlap
constexpr uint32_t WARP_EXTRA = 256 + GROUP * 32 * 4;  // nd, ni and fr after the beam's two arrays

// self-check codes, shared with the exact kernel's report
enum : unsigned { FERR_LOOP = 4u, FERR_BAD_ID = 8u, FERR_BEAM_RANGE = 32u };

struct ServeArgs {
    const float* x;
    uint32_t dp4;  // float4 per row
    uint32_t L;
    uint64_t off_base[16];
    uint32_t nrows[16];
    const uint64_t* off_all;
    const uint32_t* adj_all;
    const float* q;
    uint32_t nq;
    const uint32_t* beams;
    uint32_t beam, cap, out_k;
    uint32_t entry;
    const uint32_t* probes;
    uint32_t nprobe, g0;
    uint32_t* out_ids;
    float* out_d;
    uint32_t* visited;
    uint32_t words;
    uint32_t* vlist;
    uint32_t width;  // most unexpanded entries expanded together (1..4)
    uint32_t flat;               // nndFlatSrch: random seeds, no descent
    const uint32_t* flat_off;    // seeds of beam width b at flat_pool + flat_off[b]
    const uint32_t* flat_pool;
    unsigned* next_q;
    unsigned* overflow;
    unsigned long long* ncmps;
    unsigned long long* nexp;
    uint32_t spec_blocks;  // k_serve_team: prefetch the next list's rows with at most this many blocks
};

template <int M>
__device__ __forceinline__ float term(float a, float b, float acc) {
    const float t = a - b;
    if (M == L2) return fmaf(t, t, acc);
    if (M == L1) return acc + fabsf(t);
    return (a != 0.f || b != 0.f) ? acc + t * t / (a + b) : acc;
}
template <int M>
__device__ __forceinline__ float part4(const float4 q, const float4 r, float acc) {
    acc = term<M>(q.x, r.x, acc);
    acc = term<M>(q.y, r.y, acc);
    acc = term<M>(q.z, r.z, acc);
    return term<M>(q.w, r.w, acc);
}

// Distances from the query (qr, spread over the warp) to the rows whose ids
// lanes 0..nf-1 hold in fid (nf <= 32, warp-uniform).  Lane j returns the
// distance of row j (0 for j >= nf).
template <int M, int QV>
__device__ __forceinline__ float warp_dists(const float4 (&qr)[QV], const float4* __restrict__ x4, uint32_t dp4,
                                            uint32_t fid, uint32_t nf, uint32_t lane) {
    constexpr int NB = QV == 1 ? 8 : (QV == 2 ? 4 : 2);  // rows in flight per lane
    if (nf <= (uint32_t)NB) {
        // few rows: one xor-shuffle reduction per row.  Its sum tree pairs
        // lanes l and l^s at width s = 16, 8, .., 1 exactly as the
        // transposing butterfly below does, so the sums are the same bits.
        float4 r[NB][QV];
#pragma unroll
        for (int b = 0; b < NB; b++) {
            const uint32_t id = __shfl_sync(FULL, fid, b);
#pragma unroll
            for (int t = 0; t < QV; t++) {
                const uint32_t c4 = lane + 32u * t;
                r[b][t] = make_float4(0.f, 0.f, 0.f, 0.f);
                if ((uint32_t)b < nf && c4 < dp4) r[b][t] = __ldg(x4 + (size_t)id * dp4 + c4);
            }
        }
        float out = 0.f;
#pragma unroll
        for (int b = 0; b < NB; b++) {
            if ((uint32_t)b < nf) {
                float sum = 0.f;
#pragma unroll
                for (int t = 0; t < QV; t++) sum = part4<M>(qr[t], r[b][t], sum);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(FULL, sum, o);
                if (lane == (uint32_t)b) out = sum;
            }
        }
        return out;
    }
    float v[32];
#pragma unroll
    for (int j = 0; j < 32; j++) v[j] = 0.f;
#pragma unroll
    for (int j0 = 0; j0 < 32; j0 += NB) {
        if ((uint32_t)j0 < nf) {
            float4 r[NB][QV];
#pragma unroll
            for (int b = 0; b < NB; b++) {
                const uint32_t id = __shfl_sync(FULL, fid, j0 + b);
#pragma unroll
                for (int t = 0; t < QV; t++) {
                    const uint32_t c4 = lane + 32u * t;
                    r[b][t] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if ((uint32_t)(j0 + b) < nf && c4 < dp4) r[b][t] = __ldg(x4 + (size_t)id * dp4 + c4);
                }
            }
#pragma unroll
            for (int b = 0; b < NB; b++)
#pragma unroll
                for (int t = 0; t < QV; t++) v[j0 + b] = part4<M>(qr[t], r[b][t], v[j0 + b]);
        }
    }
    // transposing butterfly: after the level of width s, v[i] holds the
    // partial sum of distance (lane's upper bits) + i over 2x more lanes
#pragma unroll
    for (int s = 16; s >= 1; s >>= 1) {
        const bool up = (lane & s) != 0;
#pragma unroll
        for (int i = 0; i < s; i++) {
            const float send = up ? v[i] : v[i + s];
            const float keep = up ? v[i + s] : v[i];
            v[i] = keep + __shfl_xor_sync(FULL, send, s);
        }
    }
    return v[0];
}

// The same distances, NB rows at a time from load to sum: 40 registers fewer,
// so that seven CTAs fit on an SM, for a longer chain per batch (see k_serve).
template <int M, int QV>
__device__ __forceinline__ float warp_dists_short(const float4 (&qr)[QV], const float4* __restrict__ x4, uint32_t dp4,
                                                  uint32_t fid, uint32_t nf, uint32_t lane) {
    constexpr uint32_t NB = QV == 1 ? 8 : (QV == 2 ? 4 : 2);  // rows in flight per lane
    constexpr uint32_t PER = 32 / NB;                         // lanes b PER .. end with row b's sum
    float out = 0.f;
#pragma unroll 1
    for (uint32_t j0 = 0; j0 < nf; j0 += NB) {
        float4 r[NB][QV];
#pragma unroll
        for (uint32_t b = 0; b < NB; b++) {
            const uint32_t id = __shfl_sync(FULL, fid, (j0 + b) & 31);
#pragma unroll
            for (int t = 0; t < QV; t++) {
                const uint32_t c4 = lane + 32u * t;
                r[b][t] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (j0 + b < nf && c4 < dp4) r[b][t] = __ldg(x4 + (size_t)id * dp4 + c4);
            }
        }
        float v[NB];
#pragma unroll
        for (uint32_t b = 0; b < NB; b++) {
            v[b] = 0.f;
#pragma unroll
            for (int t = 0; t < QV; t++) v[b] = part4<M>(qr[t], r[b][t], v[b]);
        }
        uint32_t s = 16;
#pragma unroll
        for (uint32_t n = NB / 2; n >= 1; n >>= 1, s >>= 1) {
            const bool up = (lane & s) != 0;
#pragma unroll
            for (uint32_t i = 0; i < n; i++) {
                const float send = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
                v[i] = keep + __shfl_xor_sync(FULL, send, s);
            }
        }
#pragma unroll
        for (; s >= 1; s >>= 1) v[0] += __shfl_xor_sync(FULL, v[0], s);
        const float mine = __shfl_sync(FULL, v[0], ((lane - j0) & (NB - 1)) * PER);
        if (lane >= j0 && lane < j0 + NB && lane < nf) out = mine;
    }
    return out;
}

// NaN distances (of queries or rows with NaN, or infinities that cancel)
// count as infinite: comparisons of NaN would give the lanes different
// minima and several new entries the same place in the beam, others none.
__device__ __forceinline__ float ordered(float d) { return d == d ? d : INFINITY; }

__device__ __forceinline__ bool key_less(float da, uint32_t ia, float db, uint32_t ib) {
    return da < db || (da == db && ia < ib);
}

// Smallest d over lanes < valid, ties to the lowest lane.
__device__ __forceinline__ void warp_argmin(float d, uint32_t valid, uint32_t lane, float& md, uint32_t& ml) {
    float m = lane < valid ? d : INFINITY;
    uint32_t l = lane < valid ? lane : 32u;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float om = __shfl_xor_sync(FULL, m, o);
        const uint32_t ol = __shfl_xor_sync(FULL, l, o);
        if (om < m || (om == m && ol < l)) {
            m = om;
            l = ol;
        }
    }
    md = m;
    ml = l;
}

// Bitonic sort of one (d, id) pair per lane over lanes [0, w), w a power of
// two (warp-uniform); ascending by (d, id).  Lanes >= w are left as they are.
__device__ __forceinline__ void warp_sort(float& d, uint32_t& id, uint32_t lane, uint32_t w) {
#pragma unroll
    for (uint32_t k = 2; k <= 32; k <<= 1) {
        if (k > w) break;
#pragma unroll
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            const float od = __shfl_xor_sync(FULL, d, j);
            const uint32_t oi = __shfl_xor_sync(FULL, id, j);
            const bool asc = (lane & k) == 0 || k == w;
            const bool low = (lane & j) == 0;
            const bool other_less = key_less(od, oi, d, id);
            const bool other_more = key_less(d, id, od, oi);
            if ((low == asc) ? other_less : other_more) {
                d = od;
                id = oi;
            }
        }
    }
}

__device__ __forceinline__ void prefetch_l1(const void* p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// Bound: memory latency of a step's chain (offsets, list ids, visited set,
// rows) at the warps that are resident.  Two forms, the same steps and sums:
// DENSE, for batches of several queries per resident warp: seven CTAs per SM
// (72 registers: the rows of a list summed eight at a time, prefetched into L2
// when their ids are known); otherwise five CTAs (96 registers, 32 rows summed
// together), whose single query is shorter.  Both spill (bytes stored: 96, 148
// and 248 by row length for L2 and L1, 168 to 344 for chi-square; dense 48 to
// 104, 104 to 268); the line between them is dense_queries.  At 1M rows the 28
// warps' bitmaps (518 MB, allocated and cleared by an index's first batch) gain
// 3 to 7 %, not worth it: so at most DENSE_SCRATCH of them and their lists.  A
// hash table per query instead of a bitmap there took 1.5 times as long.
template <int M, int QV, bool DENSE>
__global__ void __launch_bounds__(FW * 32, DENSE ? 7 : 5) k_serve(ServeArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    const uint32_t w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t slot = blockIdx.x * FW + w;
    unsigned char* base = smem + (size_t)w * ((size_t)a.cap * 8 + WARP_EXTRA);
    float* bd = reinterpret_cast<float*>(base);
    uint32_t* bi = reinterpret_cast<uint32_t*>(bd + a.cap);
    float* nd = reinterpret_cast<float*>(bi + a.cap);
    uint32_t* ni = reinterpret_cast<uint32_t*>(nd + 32);
    uint32_t* fr = ni + 32;  // fresh ids of one group of a step
    uint32_t* vis = a.visited + (size_t)slot * a.words;
    uint32_t* vl = a.vlist + (size_t)slot * FVCAP;
    const float4* x4 = reinterpret_cast<const float4*>(a.x);
    const uint32_t nlast = a.nrows[a.L - 1];
    auto dists = [](const float4(&qr)[QV], const float4* x, uint32_t dp4, uint32_t fid, uint32_t nf, uint32_t lane) {
        return ordered(DENSE ? warp_dists_short<M, QV>(qr, x, dp4, fid, nf, lane)
                             : warp_dists<M, QV>(qr, x, dp4, fid, nf, lane));
    };
    unsigned long long cmps = 0, nexp = 0;
    for (;;) {
        uint32_t qi = 0;
        if (lane == 0) qi = atomicAdd(a.next_q, 1u);
        qi = __shfl_sync(FULL, qi, 0);
        if (qi >= a.nq) break;
        uint32_t ef = a.beams ? a.beams[qi] : a.beam;
        if (ef < a.out_k || ef > a.cap) {
            if (lane == 0) atomicOr(a.overflow, FERR_BEAM_RANGE);
            ef = min(max(ef, a.out_k), a.cap);
        }
        // expansions per step: wide beams take up to a.width, narrow ones 1
        const uint32_t width = max(1u, min(a.width, ef / 64));
        float4 qr[QV];
#pragma unroll
        for (int t = 0; t < QV; t++) {
            const uint32_t c4 = lane + 32u * t;
            qr[t] = c4 < a.dp4 ? __ldg(reinterpret_cast<const float4*>(a.q) + (size_t)qi * a.dp4 + c4)
                               : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        // entry
        uint32_t cur = 0, g0;
        float cur_d = 0.f;
        if (a.flat) {
            g0 = a.L - 1;  // nndFlatSrch: no descent; the seeds start the beam
        } else if (a.probes) {
            g0 = a.g0;
            uint32_t pid = 0;
            if (lane < a.nprobe) {
                pid = a.probes[(size_t)qi * a.nprobe + lane];
                if (pid >= a.nrows[g0]) {
                    atomicOr(a.overflow, FERR_BAD_ID);
                    pid = 0;
                }
            }
            const float pd = dists(qr, x4, a.dp4, pid, a.nprobe, lane);
            uint32_t l;
            warp_argmin(pd, a.nprobe, lane, cur_d, l);
            cur = __shfl_sync(FULL, pid, l & 31);
            cmps += a.nprobe;
        } else {
            g0 = 0;
            cur = a.entry;
            cur_d = __shfl_sync(FULL, dists(qr, x4, a.dp4, cur, 1, lane), 0);
            cmps++;
        }
        // greedy descent (lysearch.cpp:397-420); upper-layer ids were checked
        // against their layers when the index was made
        for (uint32_t g = g0; g + 1 < a.L; g++) {
            const uint64_t* off = a.off_all + a.off_base[g];
            uint32_t moves = 0;
            for (;;) {
                if (cur >= a.nrows[g] || ++moves > a.nrows[g]) {
                    if (lane == 0) atomicOr(a.overflow, cur >= a.nrows[g] ? FERR_BAD_ID : FERR_LOOP);
                    cur = 0;
                    break;
                }
                const uint64_t b = off[cur], e = off[cur + 1];
                float best = cur_d;
                uint32_t bid = cur;
                for (uint64_t c0 = b; c0 < e; c0 += 32) {
                    const uint32_t cnt = (uint32_t)(e - c0 < 32 ? e - c0 : 32);
                    const uint32_t nn = lane < cnt ? a.adj_all[c0 + lane] : 0u;
                    const float dd = dists(qr, x4, a.dp4, nn, cnt, lane);
                    cmps += cnt;
                    float md;
                    uint32_t ml;
                    warp_argmin(dd, cnt, lane, md, ml);
                    const uint32_t mid = __shfl_sync(FULL, nn, ml & 31);
                    if (md < best) {
                        best = md;
                        bid = mid;
                    }
                }
                if (bid == cur) break;
                cur = bid;
                cur_d = best;
            }
        }
        // beam on the last layer
        const uint64_t* off = a.off_all + a.off_base[a.L - 1];
        uint32_t m = 0, p = 0, nvis = 0;
        // Offers the fresh rows whose ids lanes [0, nf) hold: distances, the
        // ones below the worst entry of a full beam sorted by a bitonic
        // network over those lanes and merged in place -- entries before the
        // first new one keep their slots.
        auto offer = [&](uint32_t fid, uint32_t nf) {
            cmps += nf;
            const float dd = dists(qr, x4, a.dp4, fid, nf, lane);
            bool acc = lane < nf;
            if (m >= ef) acc = acc && key_less(dd, fid, bd[m - 1], bi[m - 1] & IDM);
            const uint32_t nk = __popc(__ballot_sync(FULL, acc));
            if (nk == 0) return;
            float kd = acc ? dd : INFINITY;
            uint32_t kid = acc ? fid : 0xffffffffu;
            uint32_t w = 1;
            while (w < nf) w <<= 1;
            warp_sort(kd, kid, lane, w);
            __syncwarp();
            nd[lane] = kd;
            ni[lane] = kid;
            const uint32_t m2 = min(ef, m + nk);
            uint32_t npos = 0;
            if (lane < nk) {
                uint32_t lo = 0, hi = m;
                while (lo < hi) {
                    const uint32_t md = (lo + hi) >> 1;
                    if (key_less(bd[md], bi[md] & IDM, kd, kid)) lo = md + 1;
                    else hi = md;
                }
                npos = lane + lo;
            }
            const uint32_t lo0 = __shfl_sync(FULL, npos, 0);
            __syncwarp();
            // entries from lo0 on move up by the number of new entries before
            // them, 32 at a time from the last: a chunk's places lie at or after
            // its own, so the chunks still to come are intact
            for (uint32_t s0 = m > lo0 ? lo0 + ((m - lo0 - 1) & ~31u) : 0u, more = m > lo0; more; s0 -= 32) {
                const uint32_t i = s0 + lane;
                float d0 = 0.f;
                uint32_t i0 = 0;
                if (i < m) {
                    d0 = bd[i];
                    i0 = bi[i];
                }
                __syncwarp();
                if (i < m) {
                    uint32_t lo = 0, hi = nk;
                    while (lo < hi) {
                        const uint32_t md = (lo + hi) >> 1;
                        if (key_less(nd[md], ni[md], d0, i0 & IDM)) lo = md + 1;
                        else hi = md;
                    }
                    if (i + lo < m2) {
                        bd[i + lo] = d0;
                        bi[i + lo] = i0;
                    }
                }
                more = s0 > lo0;
            }
            if (lane < nk && npos < m2) {
                bd[npos] = kd;
                bi[npos] = kid;
            }
            __syncwarp();
            m = m2;
            if (lo0 < p) p = lo0;
        };
        if (a.flat) {
            // nndFlatSrch (lysearch.cpp:455-472): the beam's getRndSds seeds
            const uint32_t* sd = a.flat_pool + a.flat_off[ef];
            for (uint32_t c0 = 0; c0 < ef; c0 += 32) {
                const uint32_t cnt = min(32u, ef - c0);
                uint32_t id = 0;
                if (lane < cnt) {
                    id = sd[c0 + lane];
                    atomicOr(&vis[id >> 5], 1u << (id & 31));
                    if (nvis + lane < FVCAP) vl[nvis + lane] = id;
                }
                nvis += cnt;
                offer(id, cnt);
            }
        } else if (cur < nlast) {
            if (lane == 0) {
                bd[0] = cur_d;
                bi[0] = cur;
                atomicOr(&vis[cur >> 5], 1u << (cur & 31));
                vl[0] = cur;
            }
            m = 1;
            nvis = 1;
        } else if (lane == 0) {
            atomicOr(a.overflow, FERR_BAD_ID);
        }
        __syncwarp();
        uint32_t expansions = 0;
        for (;;) {
            __syncwarp();  // the expanded marks and the last merge are visible
            // the first `width` unexpanded entries; lane e keeps the e-th one
            uint32_t ne = 0, mine = 0, mypos = 0, last = 0;
            for (uint32_t s0 = p; s0 < m && ne < width; s0 += 32) {
                unsigned bal = __ballot_sync(FULL, s0 + lane < m && !(bi[s0 + lane] & EXP_BIT));
                while (bal && ne < width) {
                    last = s0 + __ffs(bal) - 1;
                    bal &= bal - 1;
                    if (lane == ne) {
                        mine = bi[last] & IDM;
                        mypos = last;
                    }
                    ne++;
                }
            }
            if (ne == 0) break;
            expansions += ne;
            if (expansions > nlast) {
                if (lane == 0) atomicOr(a.overflow, FERR_LOOP);
                break;
            }
            p = last + 1;
            __syncwarp();
            if (lane < ne) bi[mypos] = mine | EXP_BIT;
            nexp += ne;
            // the selected nodes' lists, read as one sequence of `total` ids:
            // entry t belongs to list e when end_{e-1} <= t < end_e
            uint64_t lb = 0, le = 0;
            if (lane < ne) {
                lb = off[mine];
                le = off[mine + 1];
            }
            const uint32_t len = (uint32_t)(le - lb);
            uint32_t pre = len;
#pragma unroll
            for (int o = 1; o < 4; o <<= 1) {
                const uint32_t v = __shfl_up_sync(FULL, pre, o);
                if (lane >= (uint32_t)o) pre += v;
            }
            const uint32_t end0 = __shfl_sync(FULL, pre, 0), end1 = __shfl_sync(FULL, pre, 1),
                           end2 = __shfl_sync(FULL, pre, 2), total = __shfl_sync(FULL, pre, 3);
            const uint64_t base_l = lb - (pre - len);  // list e: adjacency index base_e + t
            const uint64_t base0 = __shfl_sync(FULL, base_l, 0), base1 = __shfl_sync(FULL, base_l, 1),
                           base2 = __shfl_sync(FULL, base_l, 2), base3 = __shfl_sync(FULL, base_l, 3);
            // the step's ids GROUP x 32 at a time: every list load, then every
            // visited-bit atomic, is in flight at once; the fresh ids are
            // gathered in list order and offered 32 at a time (the beam after
            // a step is the best of the union whatever the order of offers)
            for (uint32_t t0 = 0; t0 < total; t0 += 32 * GROUP) {
                uint32_t nn[GROUP];
                bool fresh[GROUP];
#pragma unroll
                for (uint32_t c = 0; c < GROUP; c++) {
                    const uint32_t t = t0 + 32 * c + lane;
                    nn[c] = 0;
                    if (t < total) {
                        const uint64_t bs = t < end0 ? base0 : (t < end1 ? base1 : (t < end2 ? base2 : base3));
                        nn[c] = a.adj_all[bs + t];
                    }
                }
#pragma unroll
                for (uint32_t c = 0; c < GROUP; c++) {
                    fresh[c] = false;
                    if (t0 + 32 * c + lane < total) {
                        const uint32_t old = atomicOr(&vis[nn[c] >> 5], 1u << (nn[c] & 31));
                        fresh[c] = !(old & (1u << (nn[c] & 31)));
                    }
                }
                uint32_t nf = 0;
                __syncwarp();  // the last offer() has finished with fr
#pragma unroll
                for (uint32_t c = 0; c < GROUP; c++) {
                    const unsigned fb = __ballot_sync(FULL, fresh[c]);
                    if (fresh[c]) {
                        const uint32_t r = nf + __popc(fb & ((1u << lane) - 1u));
                        if (DENSE)
                            for (uint32_t t = 0; t < a.dp4; t += 8) prefetch_l2(x4 + (size_t)nn[c] * a.dp4 + t);
                        fr[r] = nn[c];
                        if (nvis + r < FVCAP) vl[nvis + r] = nn[c];
                    }
                    nf += __popc(fb);
                }
                nvis += nf;
                __syncwarp();
                for (uint32_t f0 = 0; f0 < nf; f0 += 32) {
                    const uint32_t cnt = min(32u, nf - f0);
                    const uint32_t fid = lane < cnt ? fr[f0 + lane] : 0u;
                    offer(fid, cnt);
                }
            }
        }
        // results: the first out_k entries
        for (uint32_t t = lane; t < a.out_k; t += 32) {
            const size_t o = (size_t)qi * a.out_k + t;
            a.out_ids[o] = t < m ? (bi[t] & IDM) : 0xffffffffu;
            if (a.out_d) a.out_d[o] = t < m ? bd[t] : 0.f;
        }
        // clear this query's visited bits
        if (nvis <= FVCAP) {
            for (uint32_t t = lane; t < nvis; t += 32) {
                const uint32_t id = vl[t];
                atomicAnd(&vis[id >> 5], ~(1u << (id & 31)));
            }
        } else {
            for (uint32_t t = lane; t < a.words; t += 32) vis[t] = 0;
        }
        __syncwarp();
    }
    for (int o = 16; o > 0; o >>= 1) cmps += __shfl_xor_sync(FULL, cmps, o);
    if (lane == 0) {
        atomicAdd(a.ncmps, cmps / 32);
        atomicAdd(a.nexp, nexp);
    }
}

// A few queries: a block per query (k_serve_team).  The steps, the beam and
// the counts are k_serve's; what a step waits for is shared or taken off the
// chain, since one warp alone spends a step of 20 fresh rows in three
// dependent batches of row reads and two round trips to L2 for the offsets,
// the list and the visited bits:
//   - warp 0 leads; a batch of up to 32 rows is measured by the four warps at
//     once, eight rows each (two block barriers a batch);
//   - the visited bitmap lies in shared memory (cleared per query);
//   - the helpers prefetch what later steps read: the fresh rows' offsets and
//     lists, and (no more blocks than SMs) the rows of the list that is
//     expanded next if no nearer entry turns up;
//   - accepted rows are placed by rank (one shuffle pair per accepted row)
//     instead of a 15-stage sort.
// Sums have the same tree as warp_dists', so the results are the same bits.
// Bound: the latency of the leader's chain, 4,900 cycles a step of which the
// row reads are 1,900 (2,600 without the prefetched rows).  Beam 64,
// 100,000 x 128 rows, device time against k_serve's: 1 query 250 -> 155 us,
// 148 queries 415 -> 239, 592 queries 489 -> 288; faster as long as every
// query has a resident block (740 here: 472 -> 296), which is the rule that
// picks it.  At 1, 148 and 700 queries, beams 16 to 256, of k_serve's time:
// L2 0.52 to 0.82, L1 0.52 to 0.82, chi-square 0.37 to 0.65.  The beam in
// registers (up to 192 entries) against shared memory: 177 -> 155 us.
constexpr int TEAM = 4;
constexpr uint32_t TEAM_MOST = 16;  // blocks an SM: 64 warps

// Distances to rows [first, first + 8) of the cnt <= 32 ids that the lanes
// hold, into out[0, 8) (shared memory).  NB rows at a time are summed by a
// transposing butterfly (NB - 1 + 5 - log2 NB shuffles).
template <int M, int QV>
__device__ __forceinline__ void team_rows(const float4 (&qr)[QV], const float4* __restrict__ x4, uint32_t dp4,
                                          uint32_t fid, uint32_t first, uint32_t cnt, uint32_t lane, float* out) {
    constexpr uint32_t NB = QV == 1 ? 8 : (QV == 2 ? 4 : 2);  // rows in flight per lane
#pragma unroll
    for (uint32_t b0 = 0; b0 < 8; b0 += NB) {
        if (first + b0 >= cnt) break;
        float4 r[NB][QV];
#pragma unroll
        for (uint32_t b = 0; b < NB; b++) {
            const uint32_t id = __shfl_sync(FULL, fid, (first + b0 + b) & 31);
#pragma unroll
            for (int t = 0; t < QV; t++) {
                const uint32_t c4 = lane + 32u * t;
                r[b][t] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (first + b0 + b < cnt && c4 < dp4) r[b][t] = __ldg(x4 + (size_t)id * dp4 + c4);
            }
        }
        float v[NB];
#pragma unroll
        for (uint32_t b = 0; b < NB; b++) {
            v[b] = 0.f;
#pragma unroll
            for (int t = 0; t < QV; t++) v[b] = part4<M>(qr[t], r[b][t], v[b]);
        }
        uint32_t s = 16;
#pragma unroll
        for (uint32_t n = NB / 2; n >= 1; n >>= 1, s >>= 1) {
            const bool up = (lane & s) != 0;
#pragma unroll
            for (uint32_t i = 0; i < n; i++) {
                const float send = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
                v[i] = keep + __shfl_xor_sync(FULL, send, s);
            }
        }
#pragma unroll
        for (; s >= 1; s >>= 1) v[0] += __shfl_xor_sync(FULL, v[0], s);
        constexpr uint32_t PER = 32 / NB;  // lanes b PER .. hold row b
        if ((lane & (PER - 1)) == 0) out[b0 + lane / PER] = v[0];
    }
}

__host__ __device__ constexpr size_t team_words(uint32_t words) { return ((size_t)words + 3) & ~(size_t)3; }
__host__ __device__ constexpr size_t team_smem(uint32_t words, uint32_t cap) {
    return (team_words(words) + (size_t)cap * 4 + 4 * 32 + GROUP * 32 + 8) * 4;
}

// A batch handed to the helpers; cnt 0: the query is done.
struct TeamCmd {
    uint32_t cnt, next;  // ids of the batch; entry likely expanded next (or ~0)
};

// ER > 0: the beam (at most 32 ER entries) in the leader's registers, entry i
// in slot i / 32 of lane i % 32; 0: in shared memory, placed by binary search.
template <int M, int QV, int ER>
__global__ void __launch_bounds__(TEAM * 32) k_serve_team(ServeArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    const uint32_t tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    uint32_t* vis = reinterpret_cast<uint32_t*>(smem);
    float* bd = reinterpret_cast<float*>(vis + team_words(a.words));
    uint32_t* bi = reinterpret_cast<uint32_t*>(bd + a.cap);
    float* td = reinterpret_cast<float*>(bi + a.cap);
    uint32_t* ti = reinterpret_cast<uint32_t*>(td + a.cap);
    float* nd = reinterpret_cast<float*>(ti + a.cap);
    uint32_t* ni = reinterpret_cast<uint32_t*>(nd + 32);
    float* raw = reinterpret_cast<float*>(ni + 32);              // the batch's distances
    uint32_t* ids = reinterpret_cast<uint32_t*>(raw + 32);       // the batch's ids
    uint32_t* fr = ids + 32;                                     // fresh ids of a group
    TeamCmd* cmd = reinterpret_cast<TeamCmd*>(fr + GROUP * 32);  // two, in turn
    const float4* x4 = reinterpret_cast<const float4*>(a.x);
    const uint32_t nlast = a.nrows[a.L - 1];
    const uint64_t* off_last = a.off_all + a.off_base[a.L - 1];
    const bool spec = gridDim.x <= a.spec_blocks;
    unsigned long long cmps = 0, nexp = 0;
    for (uint32_t qi = blockIdx.x; qi < a.nq; qi += gridDim.x) {
        for (uint32_t i = tid; i < team_words(a.words) / 4; i += TEAM * 32)
            reinterpret_cast<uint4*>(vis)[i] = make_uint4(0u, 0u, 0u, 0u);
        float4 qr[QV];
#pragma unroll
        for (int t = 0; t < QV; t++) {
            const uint32_t c4 = lane + 32u * t;
            qr[t] = c4 < a.dp4 ? __ldg(reinterpret_cast<const float4*>(a.q) + (size_t)qi * a.dp4 + c4)
                               : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        __syncthreads();  // the bitmap is clear
        uint32_t turn = 0;
        if (w > 0) {  // helpers
            for (;; turn ^= 1) {
                __syncthreads();  // a batch is posted
                const TeamCmd c = cmd[turn];
                if (c.cnt == 0) break;
                const uint32_t fid = lane < c.cnt ? ids[lane] : 0u;
                team_rows<M, QV>(qr, x4, a.dp4, fid, 8 * w, c.cnt, lane, raw + 8 * w);
                __syncthreads();  // the batch is measured
                if (w == TEAM - 1) {
                    if (lane < c.cnt && fid < nlast) {
                        const uint64_t b = off_last[fid], e = off_last[fid + 1];
                        for (uint64_t t = b; t < e; t += 32) prefetch_l1(a.adj_all + t);
                        if (e > b) prefetch_l1(a.adj_all + e - 1);
                    }
                } else if (spec) {
                    // the rows of the list that the next step reads, of one of
                    // two entries: the first open one, or the nearest of this batch
                    uint32_t cand = c.next;
                    if (w == 1) {
                        const uint32_t u = lane < c.cnt ? __float_as_uint(raw[lane]) : 0u;
                        const uint32_t key = lane < c.cnt ? (u >> 31 ? ~u : u | 0x80000000u) : 0xffffffffu;
                        const unsigned at = __ballot_sync(FULL, key == __reduce_min_sync(FULL, key));
                        cand = __shfl_sync(FULL, fid, __ffs(at) - 1);
                    }
                    if (cand < nlast) {
                        const uint64_t b = off_last[cand], e = off_last[cand + 1];
                        if (b + lane < e) {
                            const uint32_t id = a.adj_all[b + lane];
                            if (!(vis[id >> 5] >> (id & 31) & 1u)) {  // a hint: the leader may be setting bits
                                const float4* r = x4 + (size_t)id * a.dp4;
                                for (uint32_t t = 0; t < a.dp4; t += 8) prefetch_l1(r + t);
                            }
                        }
                    }
                }
            }
            __syncthreads();  // the results are out
            continue;
        }
        // leader
        uint32_t ef = a.beams ? a.beams[qi] : a.beam;
        if (ef < a.out_k || ef > a.cap) {
            if (lane == 0) atomicOr(a.overflow, FERR_BEAM_RANGE);
            ef = min(max(ef, a.out_k), a.cap);
        }
        const uint32_t width = max(1u, min(a.width, ef / 64));
        // distances of the cnt <= 32 ids in the lanes
        auto dists = [&](uint32_t fid, uint32_t cnt, uint32_t next) -> float {
            if (lane < cnt) ids[lane] = fid;
            if (lane == 0) cmd[turn] = TeamCmd{cnt, next};
            turn ^= 1;
            __syncthreads();
            team_rows<M, QV>(qr, x4, a.dp4, fid, 0, cnt, lane, raw);
            __syncthreads();
            return ordered(raw[lane]);
        };
        uint32_t cur = 0, g0;
        float cur_d = 0.f;
        if (a.flat) {
            g0 = a.L - 1;
        } else if (a.probes) {
            g0 = a.g0;
            uint32_t pid = 0;
            if (lane < a.nprobe) {
                pid = a.probes[(size_t)qi * a.nprobe + lane];
                if (pid >= a.nrows[g0]) {
                    atomicOr(a.overflow, FERR_BAD_ID);
                    pid = 0;
                }
            }
            uint32_t l;
            warp_argmin(dists(pid, a.nprobe, ~0u), a.nprobe, lane, cur_d, l);
            cur = __shfl_sync(FULL, pid, l & 31);
            cmps += a.nprobe;
        } else {
            g0 = 0;
            cur = a.entry;
            cur_d = __shfl_sync(FULL, dists(cur, 1, ~0u), 0);
            cmps++;
        }
        // greedy descent, as k_serve
        for (uint32_t g = g0; g + 1 < a.L; g++) {
            const uint64_t* off = a.off_all + a.off_base[g];
            uint32_t moves = 0;
            for (;;) {
                if (cur >= a.nrows[g] || ++moves > a.nrows[g]) {
                    if (lane == 0) atomicOr(a.overflow, cur >= a.nrows[g] ? FERR_BAD_ID : FERR_LOOP);
                    cur = 0;
                    break;
                }
                const uint64_t b = off[cur], e = off[cur + 1];
                float best = cur_d;
                uint32_t bid = cur;
                for (uint64_t c0 = b; c0 < e; c0 += 32) {
                    const uint32_t cnt = (uint32_t)(e - c0 < 32 ? e - c0 : 32);
                    const uint32_t nn = lane < cnt ? a.adj_all[c0 + lane] : 0u;
                    if (lane < cnt) prefetch_l1(off + nn);
                    const float dd = dists(nn, cnt, ~0u);
                    cmps += cnt;
                    float md;
                    uint32_t ml;
                    warp_argmin(dd, cnt, lane, md, ml);
                    const uint32_t mid = __shfl_sync(FULL, nn, ml & 31);
                    if (md < best) {
                        best = md;
                        bid = mid;
                    }
                }
                if (bid == cur) break;
                cur = bid;
                cur_d = best;
            }
        }
        uint32_t m = 0, p = 0;
        constexpr int ES = ER ? ER : 1;
        float rd[ES];
        uint32_t ri[ES];
#pragma unroll
        for (int r = 0; r < ES; r++) {
            rd[r] = INFINITY;
            ri[r] = 0xffffffffu;
        }
        // the first unexpanded entry from s0 on (its position; m: none)
        auto first_open = [&](uint32_t s0) -> uint32_t {
            if (ER) {
                uint32_t at = m;
#pragma unroll
                for (int r = ES - 1; r >= 0; r--) {
                    const uint32_t i = 32u * r + lane;
                    const unsigned bal = __ballot_sync(FULL, i >= s0 && i < m && !(ri[r] & EXP_BIT));
                    if (bal) at = 32u * r + __ffs(bal) - 1;
                }
                return at;
            }
            for (; s0 < m; s0 += 32) {
                const unsigned bal = __ballot_sync(FULL, s0 + lane < m && !(bi[s0 + lane] & EXP_BIT));
                if (bal) return s0 + __ffs(bal) - 1;
            }
            return m;
        };
        // id word of entry `at` < m
        auto id_at = [&](uint32_t at) -> uint32_t {
            if (!ER) return bi[at];
            uint32_t v = ri[0];
#pragma unroll
            for (int r = 1; r < ES; r++)
                if ((at >> 5) == (uint32_t)r) v = ri[r];
            return __shfl_sync(FULL, v, at & 31);
        };
        auto dist_at = [&](uint32_t at) -> float {
            if (!ER) return bd[at];
            float v = rd[0];
#pragma unroll
            for (int r = 1; r < ES; r++)
                if ((at >> 5) == (uint32_t)r) v = rd[r];
            return __shfl_sync(FULL, v, at & 31);
        };
        auto mark = [&](uint32_t at) {
            if (ER) {
#pragma unroll
                for (int r = 0; r < ES; r++)
                    if (at == 32u * r + lane) ri[r] |= EXP_BIT;
            } else {
                __syncwarp();
                if (lane == 0) bi[at] |= EXP_BIT;
                __syncwarp();
            }
        };
        // k_serve's offer; next: see TeamCmd
        auto offer = [&](uint32_t fid, uint32_t nf, uint32_t next) {
            cmps += nf;
            float wd = INFINITY;
            uint32_t wi = 0xffffffffu;
            if (m >= ef) {
                wd = dist_at(m - 1);
                wi = id_at(m - 1) & IDM;
            }
            const float dd = dists(fid, nf, next);
            const bool acc = lane < nf && (m < ef || key_less(dd, fid, wd, wi));
            const unsigned am = __ballot_sync(FULL, acc);
            const uint32_t nk = __popc(am);
            if (nk == 0) return;
            const uint32_t m2 = min(ef, m + nk);
            uint32_t rank = 0;
            if (ER) {
                // every accepted row against the beam and the other rows: its
                // place, and how far each entry moves up
                uint32_t place = 0, move[ES];
#pragma unroll
                for (int r = 0; r < ES; r++) move[r] = 0;
#pragma unroll 2
                for (unsigned q = am; q; q &= q - 1) {
                    const int j = __ffs(q) - 1;
                    const float od = __shfl_sync(FULL, dd, j);
                    const uint32_t oi = __shfl_sync(FULL, fid, j);
                    rank += key_less(od, oi, dd, fid) || (od == dd && oi == fid && j < (int)lane);
                    uint32_t before = 0;
#pragma unroll
                    for (int r = 0; r < ES; r++) {
                        const bool less = key_less(rd[r], ri[r] & IDM, od, oi);
                        before += __popc(__ballot_sync(FULL, less));
                        move[r] += !less;
                    }
                    if ((int)lane == j) place = before;
                }
#pragma unroll
                for (int r = 0; r < ES; r++) {
                    const uint32_t i = 32u * r + lane, to = i + move[r];
                    if (i < m && to < m2) {
                        bd[to] = rd[r];
                        bi[to] = ri[r];
                    }
                }
                if (acc && place + rank < m2) {
                    bd[place + rank] = dd;
                    bi[place + rank] = fid;
                }
                __syncwarp();
#pragma unroll
                for (int r = 0; r < ES; r++) {
                    const uint32_t i = 32u * r + lane;
                    if (i < m2) {
                        rd[r] = bd[i];
                        ri[r] = bi[i];
                    }
                }
                __syncwarp();
                m = m2;
                return;
            }
            for (unsigned r = am; r; r &= r - 1) {
                const int j = __ffs(r) - 1;
                const float od = __shfl_sync(FULL, dd, j);
                const uint32_t oi = __shfl_sync(FULL, fid, j);
                rank += key_less(od, oi, dd, fid) || (od == dd && oi == fid && j < (int)lane);
            }
            uint32_t npos = 0xffffffffu;
            if (acc) {
                uint32_t lo = 0, hi = m;
                while (lo < hi) {
                    const uint32_t md = (lo + hi) >> 1;
                    const float v = bd[md];
                    if (v < dd || (v == dd && (bi[md] & IDM) < fid)) lo = md + 1;
                    else hi = md;
                }
                npos = rank + lo;
                nd[rank] = dd;
                ni[rank] = fid;
            }
            const uint32_t lo0 = __reduce_min_sync(FULL, npos);
            for (uint32_t i = lo0 + lane; i < m; i += 32) {
                td[i - lo0] = bd[i];
                ti[i - lo0] = bi[i];
            }
            __syncwarp();
            for (uint32_t i = lo0 + lane; i < m; i += 32) {
                const float d0 = td[i - lo0];
                const uint32_t i0 = ti[i - lo0];
                uint32_t lo = 0, hi = nk;
                while (lo < hi) {
                    const uint32_t md = (lo + hi) >> 1;
                    if (key_less(nd[md], ni[md], d0, i0 & IDM)) lo = md + 1;
                    else hi = md;
                }
                if (i + lo < m2) {
                    bd[i + lo] = d0;
                    bi[i + lo] = i0;
                }
            }
            if (acc && npos < m2) {
                bd[npos] = dd;
                bi[npos] = fid;
            }
            __syncwarp();
            m = m2;
            if (lo0 < p) p = lo0;
        };
        if (a.flat) {
            const uint32_t* sd = a.flat_pool + a.flat_off[ef];
            for (uint32_t c0 = 0; c0 < ef; c0 += 32) {
                const uint32_t cnt = min(32u, ef - c0);
                uint32_t id = 0;
                if (lane < cnt) {
                    id = sd[c0 + lane];
                    atomicOr(&vis[id >> 5], 1u << (id & 31));
                }
                offer(id, cnt, ~0u);
            }
        } else if (cur < nlast) {
            if (lane == 0) {
                rd[0] = bd[0] = cur_d;
                ri[0] = bi[0] = cur;
                atomicOr(&vis[cur >> 5], 1u << (cur & 31));
            }
            m = 1;
        } else if (lane == 0) {
            atomicOr(a.overflow, FERR_BAD_ID);
        }
        uint32_t expansions = 0;
        for (;;) {
            __syncwarp();  // the last merge is visible
            // lane e: the e-th of the first `width` unexpanded entries
            uint32_t ne = 0, mine = 0, at = first_open(p);
            while (at < m) {
                const uint32_t id = id_at(at) & IDM;
                if (lane == ne) mine = id;
                mark(at);
                if (!ER) p = at + 1;
                if (++ne >= width) break;
                at = first_open(at + 1);
            }
            if (ne == 0) break;
            expansions += ne;
            if (expansions > nlast) {
                if (lane == 0) atomicOr(a.overflow, FERR_LOOP);
                break;
            }
            nexp += ne;
            uint64_t lb = 0, le = 0;
            if (lane < ne) {
                lb = off_last[mine];
                le = off_last[mine + 1];
            }
            const uint32_t open = first_open(p), next = open < m ? id_at(open) & IDM : ~0u;  // while those load
            const uint32_t len = (uint32_t)(le - lb);
            uint32_t pre = len;
            uint64_t base_l = lb;
            if (ne > 1) {
#pragma unroll
                for (int o = 1; o < 4; o <<= 1) {
                    const uint32_t v = __shfl_up_sync(FULL, pre, o);
                    if (lane >= (uint32_t)o) pre += v;
                }
                base_l = lb - (pre - len);  // list e: adjacency index base_e + t
            }
            const uint32_t total = __shfl_sync(FULL, pre, ne - 1);
            for (uint32_t t0 = 0; t0 < total; t0 += 32 * GROUP) {
                uint32_t nn[GROUP];
#pragma unroll
                for (uint32_t c = 0; c < GROUP; c++) {
                    if (t0 + 32 * c >= total) break;
                    const uint32_t t = t0 + 32 * c + lane;
                    uint64_t bs = __shfl_sync(FULL, base_l, 0);
                    for (uint32_t e = 1; e < ne; e++) {  // entry t belongs to list e when end_{e-1} <= t
                        const uint32_t end = __shfl_sync(FULL, pre, e - 1);
                        const uint64_t be = __shfl_sync(FULL, base_l, e);
                        if (t >= end) bs = be;
                    }
                    nn[c] = t < total ? a.adj_all[bs + t] : 0u;
                }
                uint32_t nf = 0;
#pragma unroll
                for (uint32_t c = 0; c < GROUP; c++) {
                    if (t0 + 32 * c >= total) break;
                    bool fresh = false;
                    if (t0 + 32 * c + lane < total) {
                        const uint32_t bit = 1u << (nn[c] & 31);
                        fresh = !(atomicOr(&vis[nn[c] >> 5], bit) & bit);
                    }
                    const unsigned fb = __ballot_sync(FULL, fresh);
                    if (fresh) {
                        fr[nf + __popc(fb & ((1u << lane) - 1u))] = nn[c];
                        prefetch_l1(off_last + nn[c]);
                    }
                    nf += __popc(fb);
                }
                __syncwarp();
                for (uint32_t f0 = 0; f0 < nf; f0 += 32) {
                    const uint32_t cnt = min(32u, nf - f0);
                    const uint32_t fid = lane < cnt ? fr[f0 + lane] : 0u;
                    offer(fid, cnt, next);
                }
                __syncwarp();
            }
        }
        if (lane == 0) cmd[turn] = TeamCmd{0, 0};
        __syncthreads();  // the helpers stop
        if (ER) {  // the marks are in the registers only; ids and distances are staged
#pragma unroll
            for (int r = 0; r < ES; r++) {
                const uint32_t i = 32u * r + lane;
                if (i < m) {
                    bd[i] = rd[r];
                    bi[i] = ri[r];
                }
            }
            __syncwarp();
        }
        for (uint32_t t = lane; t < a.out_k; t += 32) {
            const size_t o = (size_t)qi * a.out_k + t;
            a.out_ids[o] = t < m ? (bi[t] & IDM) : 0xffffffffu;
            if (a.out_d) a.out_d[o] = t < m ? bd[t] : 0.f;
        }
        __syncthreads();
    }
    if (tid == 0) {
        atomicAdd(a.ncmps, cmps);
        atomicAdd(a.nexp, nexp);
    }
}

#ifdef NNM_SERVE_FORM
using ServeFn = void (*)(ServeArgs);
template <int M>
ServeFn pick_warp(uint32_t qv, bool dense) {
    if (dense) return qv == 1 ? k_serve<M, 1, true> : (qv == 2 ? k_serve<M, 2, true> : k_serve<M, 4, true>);
    return qv == 1 ? k_serve<M, 1, false> : (qv == 2 ? k_serve<M, 2, false> : k_serve<M, 4, false>);
}
template <int M, int QV>
ServeFn pick_team_beam(uint32_t beam) {
    return beam <= 64 ? k_serve_team<M, QV, 2> : (beam <= 192 ? k_serve_team<M, QV, 6> : k_serve_team<M, QV, 0>);
}
template <int M>
ServeFn pick_team(uint32_t qv, uint32_t beam) {
    return qv == 1 ? pick_team_beam<M, 1>(beam) : (qv == 2 ? pick_team_beam<M, 2>(beam) : pick_team_beam<M, 4>(beam));
}
#else
// The dense form takes batches of more queries per SM than this (0: none).
// Wider beams visit more rows and so wait more for the bitmaps, which 28 warps
// an SM push out of the L2 sooner.  Device time, dense / not, at 8,300 to
// 18,000 queries (56 to 122 an SM; 56 is two for every dense warp):
//   rows of four float4 a lane, and chi-square: 0.17 to 0.73 from 56 on;
//   beams 16 and 64: 0.79 to 0.94 and 0.85 to 1.05 from 56 on;
//   beams 100 to 512, by the bitmaps of the dense form (rows):
//     16 MB (31,000): 0.94 to 1.08 at 56, 0.89 to 1.01 from 67 on;
//     64 MB (124,000), to beam 128: 0.98 to 1.12 at 61, 0.92 to 1.04 at 81, 0.87
//       to 0.96 from 100 on; above: 0.99 to 1.17 at 56 and 61, 0.93 to 1.07 at
//       81, 0.90 to 0.99 from 100 on;
//     above, to beam 128: 0.99 to 1.13 at 61, 0.86 to 1.05 at 88, 0.90 to 1.01
//       from 100 on; wider, one float4 a lane: 1.05 to 1.22 at 61, 0.99 to 1.05
//       at 108 and 122; two: 1.15 to 1.20 at 61, 0.95 to 0.98 at 108.
uint32_t dense_queries(int metric, uint32_t qv, uint32_t beam, size_t bitmaps) {
    if (metric == CHI2 || qv > 2 || beam <= 64) return 56;
    if (bitmaps <= (size_t)16 << 20) return 64;
    if (bitmaps <= (size_t)64 << 20) return beam <= 128 ? 72 : 100;
    return beam <= 128 || qv > 1 ? 100 : 0;
}
#endif
}  // namespace

// This file is compiled seven times: for the host side, and for the kernels of
// each form (NNM_SERVE_FORM: warp, team) and metric.  A form's kernels are a
// module of their own, so that a program's first search loads the forms it
// may run and not all 45 (its first one-query call: 28 -> 2 ms), and they
// compile side by side.
#define NNM_SERVE_NAME_(form, metric) serve_##form##_##metric
#define NNM_SERVE_NAME(form, metric) NNM_SERVE_NAME_(form, metric)
#ifdef NNM_SERVE_FORM
#define NNM_SERVE_PICK_(form) pick_##form
#define NNM_SERVE_PICK(form) NNM_SERVE_PICK_(form)
const void* NNM_SERVE_NAME(NNM_SERVE_FORM, NNM_SERVE_METRIC)(uint32_t qv, uint32_t arg) {
    return reinterpret_cast<const void*>(NNM_SERVE_PICK(NNM_SERVE_FORM)<NNM_SERVE_METRIC>(qv, arg));
}
#else
// The kernel for qv float4 a lane: arg = the dense form (warp), or the widest
// beam (team).
using ServePick = const void* (*)(uint32_t qv, uint32_t arg);
const void *serve_warp_L2(uint32_t, uint32_t), *serve_warp_L1(uint32_t, uint32_t), *serve_warp_CHI2(uint32_t, uint32_t),
    *serve_team_L2(uint32_t, uint32_t), *serve_team_L1(uint32_t, uint32_t), *serve_team_CHI2(uint32_t, uint32_t);

int index_run_fast(Ctx& ctx, IndexDev& ix, const SearchReq& r) {
    cudaStream_t st = ctx.stream;
    if (ix.dp > FAST_MAX_DP) {
        ctx.last_error = "fast search supports d <= 512";
        return 1;
    }
    const uint32_t dp4 = ix.dp / 4;
    const uint32_t qv = dp4 <= 32 ? 1 : (dp4 <= 64 ? 2 : 4);
    int nsm = 148, per_sm = 1, optin = 0;
    NNM_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, ctx.device));
    NNM_CUDA_TRY(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx.device));
    const uint32_t words = (ix.n + 31) / 32;
    // a block per query while the blocks resident at once hold them all, and
    // the visited bitmap fits in shared memory
    const ServePick pick_team = ix.metric == L2 ? serve_team_L2 : (ix.metric == L1 ? serve_team_L1 : serve_team_CHI2);
    const ServePick pick_warp = ix.metric == L2 ? serve_warp_L2 : (ix.metric == L1 ? serve_warp_L1 : serve_warp_CHI2);
    const void* fn = nullptr;
    const size_t tsmem = team_smem(words, r.beam_max);
    bool use_team = tsmem <= (size_t)optin && r.nq <= TEAM_MOST * (uint32_t)nsm;
    if (use_team) {
        const void* team = pick_team(qv, r.beam_max);
        NNM_CUDA_TRY(cudaFuncSetAttribute(team, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tsmem));
        int pt = 0;
        NNM_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&pt, team, TEAM * 32, tsmem));
        use_team = r.nq <= (uint32_t)std::max(pt, 0) * (uint32_t)nsm;
        if (use_team) fn = team;
    }
    // several queries per resident warp: the form with more warps
    const bool dense_fits = ((size_t)words + FVCAP) * 4 * DENSE_WARPS * nsm <= DENSE_SCRATCH;
    const uint32_t line = dense_queries((int)ix.metric, qv, r.beam_max, (size_t)words * 4 * DENSE_WARPS * nsm);
    const bool dense = !use_team && dense_fits && line && r.nq > line * (uint32_t)nsm;
    if (!fn) fn = pick_warp(qv, dense);
    const size_t smem = use_team ? tsmem : (size_t)FW * ((size_t)r.beam_max * 8 + WARP_EXTRA);
    uint32_t blocks = r.nq;
    if (!use_team) {
        NNM_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, FW * 32, smem);
        blocks = std::min((uint32_t)std::min(std::max(1, per_sm), 8) * (uint32_t)nsm, (r.nq + FW - 1) / FW);
        const uint32_t full = (dense_fits ? DENSE_WARPS : WARPS) / FW * (uint32_t)nsm;
        const size_t slots = (size_t)scratch_blocks(blocks, full, (uint32_t)nsm) * FW;
        if (ix.visited.bytes < slots * words * 4) {
            NNM_CUDA_TRY(ix.visited.ensure(slots * words * 4));
            NNM_CUDA_TRY(cudaMemsetAsync(ix.visited.p, 0, slots * words * 4, st));
        }
        NNM_CUDA_TRY(ix.vlist.ensure(slots * FVCAP * 4));
    }
    ServeArgs a{};
    a.x = ix.x.as<float>();
    a.dp4 = dp4;
    a.L = ix.L;
    for (uint32_t g = 0; g < ix.L; g++) {
        a.off_base[g] = ix.off_base[g];
        a.nrows[g] = ix.nrows[g];
    }
    a.off_all = ix.off.as<uint64_t>();
    a.adj_all = ix.adj.as<uint32_t>();
    a.q = r.q;
    a.nq = r.nq;
    a.beams = r.beams;
    a.beam = r.beam;
    a.cap = r.beam_max;
    a.out_k = r.out_k;
    a.entry = ix.entry;
    a.probes = r.probes;
    a.nprobe = r.nprobe;
    a.g0 = r.g0;
    a.out_ids = r.out_ids;
    a.out_d = r.out_d;
    a.visited = ix.visited.as<uint32_t>();
    a.words = words;
    a.vlist = ix.vlist.as<uint32_t>();
    a.width = ix.width;
    a.flat = r.flat;
    a.flat_off = r.flat_off;
    a.flat_pool = r.flat_pool;
    unsigned char* c = ix.ctr.as<unsigned char>();
    a.next_q = reinterpret_cast<unsigned*>(c);
    a.overflow = reinterpret_cast<unsigned*>(c + 4);
    a.ncmps = reinterpret_cast<unsigned long long*>(c + 8);
    a.nexp = reinterpret_cast<unsigned long long*>(c + 16);
    a.spec_blocks = (uint32_t)nsm;
    void* args[] = {&a};
    NNM_CUDA_TRY(cudaLaunchKernel(fn, dim3(blocks), dim3((use_team ? TEAM : FW) * 32), args, smem, st)); count_launch();
    return 0;
}
#endif

}  // namespace nnm
