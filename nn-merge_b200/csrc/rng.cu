// Reference-exact random streams.
//
// 1. std::rand() (glibc, the generator behind std::random_shuffle in
//    kgraph.cpp:139-162 and friends).  glibc's TYPE_3 generator is the
//    additive lagged-Fibonacci sequence
//        r[i] = r[i-31] + r[i-3]  (mod 2^32),   rand() #k = r[k+344] >> 1,
//    with r[0..30] from srand's Park-Miller fill and r[31..33] = r[0..2].
//    The recurrence is linear, so s[n] = r[34+n] equals sum_j c_j s[j] where
//    c = x^n mod P(x), P(x) = x^31 - x^28 - 1, coefficients mod 2^32.  Each
//    warp jumps to its own run with a product of precomputed x^(d 16^j) mod P
//    and then runs the recurrence, a lane per word: the whole stream for an
//    NN-Descent iteration is produced in parallel, with no host work.
// 2. std::mt19937 draws for the initial graphs and the cross samples
//    (Matsumoto & Nishimura, "Mersenne Twister", ACM TOMACS 1998).  The
//    recurrence x[i+624] = x[i+397] ^ f(x[i], x[i+1]) gives 227 new words at
//    a time from older ones, so one CTA runs the stream (k_mt19937); every
//    phase of a build draws from mt19937(seed), so a build generates its
//    longest phase's stream once and the others read its prefix.
#include <cstdint>
#include <cstring>
#include <random>
#include <vector>

#include "nnm_rng.h"
#include "nnm_launch.h"

namespace nnm {

namespace {
constexpr int DEG = 31;
constexpr int RUN = 16;          // blocks of 31 outputs a warp generates
constexpr int STREAM_WARPS = 8;  // warps per CTA
constexpr unsigned FULL = 0xffffffffu;

// x^(d 16^j) mod P, d = 1..15 (independent of the seed), 32 words apiece
// (the last one 0).
__device__ uint32_t g_pow16[16][15][32];

// a * b mod P, a coefficient per lane (lane 31 holds 0), mod 2^32.  Lane k
// sums the product's coefficients k (lo) and k + 32 (hi): the two need the
// same b, lane (k - i) mod 32.  The high half folds down with x^31 = x^28 +
// 1: a suffix sum of stride 3 over the coefficients 31, 32, ...
__device__ __forceinline__ uint32_t poly_mulmod_warp(uint32_t a, uint32_t b, int lane) {
    uint32_t lo = 0, hi = 0;
#pragma unroll
    for (int i = 0; i < DEG; i++) {
        const uint32_t p = __shfl_sync(FULL, a, i) * __shfl_sync(FULL, b, (lane - i) & 31);
        if (i <= lane) lo += p;
        else hi += p;
    }
    uint32_t h = __shfl_up_sync(FULL, hi, 1);
    const uint32_t t31 = __shfl_sync(FULL, lo, 31);
    if (lane == 0) h = t31;
#pragma unroll
    for (int s = 3; s < 32; s *= 2) {
        const uint32_t o = __shfl_down_sync(FULL, h, s);
        if (lane + s < 32) h += o;
    }
    const uint32_t f = __shfl_sync(FULL, h, (lane - 28) & 31);
    lo += h + (lane >= 28 ? f : 0u);
    return lane < DEG ? lo : 0u;
}

// A warp per run of 31 RUN outputs, 31 lanes a word each: a block of 31 is
// one stride-3 prefix sum over the lanes, its 124 bytes one coalesced store.
// A thread per 2,048 outputs, each with the 961-term product in registers
// and its own stores 8 KB from its neighbours', took 140 us per iteration of
// a 100,000-row build (2M draws) and 32 us at 2,000 rows, where a handful of
// threads did all the work.
__global__ void __launch_bounds__(STREAM_WARPS * 32) k_glibc_stream(int32_t* __restrict__ out, GlibcBase base,
                                                                    uint64_t first_output,
                                                                    const uint64_t* __restrict__ count_ptr,
                                                                    uint64_t count_cap) {
    __shared__ uint32_t bs[2 * DEG];
    for (uint32_t i = threadIdx.x; i < 2 * DEG; i += blockDim.x) bs[i] = base.s[i];
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const uint64_t g = (uint64_t)blockIdx.x * STREAM_WARPS + (threadIdx.x >> 5);
    uint64_t count = count_ptr ? *count_ptr : count_cap;
    if (count > count_cap) count = count_cap;
    const uint64_t k0 = g * (DEG * RUN);
    if (k0 >= count) return;
    // x^n for the s-index n of the run's first output, a hexadecimal digit at a time
    const uint64_t n = first_output + k0 + 310;
    // (n >= 310: digit 2 or a higher one is not 0); the table reads of eight
    // digits are in flight at once
    uint32_t c = lane == 0 ? 1u : 0u;
    bool one = true;
    for (int j0 = 0; j0 < 16 && (n >> (4 * j0)); j0 += 8) {
        uint32_t pw[8];
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const uint32_t d = (uint32_t)(n >> (4 * (j0 + j))) & 15u;
            pw[j] = d ? g_pow16[j0 + j][d - 1][lane] : 0u;
        }
#pragma unroll 1
        for (int j = 0; j < 8; j++) {
            const uint32_t d = (uint32_t)(n >> (4 * (j0 + j))) & 15u;
            uint32_t p = pw[0];
#pragma unroll
            for (int q = 1; q < 8; q++)
                if (q == j) p = pw[q];
            if (!d) continue;
            c = one ? p : poly_mulmod_warp(c, p, lane);
            one = false;
        }
    }
    uint32_t w = 0;
    const int m = lane < DEG ? lane : DEG - 1;
#pragma unroll
    for (int j = 0; j < DEG; j++) w += __shfl_sync(FULL, c, j) * bs[j + m];
    const int src = 28 + m % 3;
    const uint64_t end = k0 + DEG * RUN < count ? k0 + DEG * RUN : count;
    for (uint64_t pos = k0; pos < end; pos += DEG) {
        if (lane < DEG && pos + lane < end) out[pos + lane] = (int32_t)(w >> 1);
        const uint32_t last = __shfl_sync(FULL, w, src);
#pragma unroll
        for (int s = 3; s < 32; s *= 2) {
            const uint32_t o = __shfl_up_sync(FULL, w, s);
            if (lane >= s) w += o;
        }
        w += last;
    }
}

// One CTA, thread t < 227 owning word t of every round of 227.  Round r
// makes the raw words x[624 + 227 r + t] (output number 227 r + t): the
// x[i+397] operand is the thread's own word of the round before, kept in a
// register, and x[i], x[i+1] are at least two rounds old -- so two rounds run
// per barrier.  The raw words lie in a ring of 2048, where the 454 read and
// the 454 written by a pair of rounds (624 words later) never alias.  Bound:
// the latency of one pair (shared-memory loads, six dependent integer
// operations, barrier).  The host's generator and the copy it replaces left
// the GPU idle for 13 ms of a 100,000-row S-Merge of 38 ms (three phases,
// 4.3M draws in all).
constexpr uint32_t MT_N = 624, MT_STEP = 227, MT_RING = 2048;
__global__ void __launch_bounds__(256) k_mt19937(MtSeed seed, uint32_t* __restrict__ ring_io, uint64_t first_round,
                                                 uint64_t rounds, uint32_t* __restrict__ out) {
    __shared__ uint32_t ring[MT_RING];
    const uint32_t t = threadIdx.x;
    if (first_round == 0)
        for (uint32_t i = t; i < MT_N; i += blockDim.x) ring[i] = seed.x[i];
    else
        for (uint32_t i = t; i < MT_RING; i += blockDim.x) ring[i] = ring_io[i];
    __syncthreads();
    uint64_t o = first_round * MT_STEP;
    uint32_t b = (uint32_t)(o % MT_RING);  // ring position of the round's x[i]
    uint32_t v = t < MT_STEP ? ring[(b + t + 397) % MT_RING] : 0u;
    auto step = [&](uint32_t a0, uint32_t a1, uint32_t pos, uint64_t at) {
        const uint32_t y = (a0 & 0x80000000u) | (a1 & 0x7fffffffu);
        v ^= (y >> 1) ^ ((a1 & 1u) ? 0x9908b0dfu : 0u);
        ring[(pos + t + MT_N) % MT_RING] = v;
        uint32_t z = v;
        z ^= z >> 11;
        z ^= (z << 7) & 0x9d2c5680u;
        z ^= (z << 15) & 0xefc60000u;
        z ^= z >> 18;
        out[at + t] = z;
    };
    for (uint64_t r = 0; r < rounds; r += 2) {  // rounds is even
        if (t < MT_STEP) {
            const uint32_t b1 = b + MT_STEP;
            const uint32_t p0 = ring[(b + t) % MT_RING], p1 = ring[(b + t + 1) % MT_RING];
            const uint32_t q0 = ring[(b1 + t) % MT_RING], q1 = ring[(b1 + t + 1) % MT_RING];
            step(p0, p1, b, o);
            step(q0, q1, b1, o + MT_STEP);
        }
        b = (b + 2 * MT_STEP) % MT_RING;
        o += 2 * MT_STEP;
        __syncthreads();
    }
    for (uint32_t i = t; i < MT_RING; i += blockDim.x) ring_io[i] = ring[i];
}

void host_mulmod(const uint32_t* a, const uint32_t* b, uint32_t* c) {
    uint32_t t[2 * DEG - 1] = {0};
    for (int i = 0; i < DEG; i++)
        for (int j = 0; j < DEG; j++) t[i + j] += a[i] * b[j];
    for (int i = 2 * DEG - 2; i >= DEG; i--) {
        t[i - 3] += t[i];
        t[i - DEG] += t[i];
    }
    std::memcpy(c, t, sizeof(uint32_t) * DEG);
}
}  // namespace

GlibcBase glibc_base(uint32_t seed) {
    // r[0..30]: srandom_r's fill; r[31..33] = r[0..2]; s[n] = r[34+n].
    if (seed == 0) seed = 1;
    std::vector<uint32_t> r(34 + 2 * DEG);
    int32_t word = (int32_t)seed;
    r[0] = (uint32_t)word;
    for (int i = 1; i < 31; i++) {
        long hi = word / 127773, lo = word % 127773;
        word = (int32_t)(16807 * lo - 2836 * hi);
        if (word < 0) word += 2147483647;
        r[i] = (uint32_t)word;
    }
    for (int i = 31; i < 34; i++) r[i] = r[i - 31];
    for (size_t i = 34; i < r.size(); i++) r[i] = r[i - 3] + r[i - 31];
    GlibcBase b;
    for (int i = 0; i < 2 * DEG; i++) b.s[i] = r[34 + i];
    return b;
}

cudaError_t glibc_tables_init() {
    static uint32_t pw[16][15][32];
    static const bool filled = [] {
        uint32_t x[DEG] = {0};
        x[1] = 1;
        for (int j = 0; j < 16; j++) {
            uint32_t p[DEG];
            std::memcpy(p, x, sizeof(p));
            for (int d = 0; d < 15; d++) {
                std::memcpy(pw[j][d], p, sizeof(p));
                host_mulmod(pw[j][d], x, p);  // p = x^((d + 2) 16^j)
            }
            std::memcpy(x, p, sizeof(p));     // x^(16 16^j)
        }
        return true;
    }();
    (void)filled;
    return cudaMemcpyToSymbol(g_pow16, pw, sizeof(pw));
}

cudaError_t glibc_stream_generate(int32_t* out, const GlibcBase& base, uint64_t first_output,
                                  const uint64_t* d_count, uint64_t count_cap, cudaStream_t st) {
    if (count_cap == 0) return cudaSuccess;
    const uint64_t per = (uint64_t)DEG * RUN * STREAM_WARPS;
    k_glibc_stream<<<(unsigned)((count_cap + per - 1) / per), STREAM_WARPS * 32, 0, st>>>(out, base, first_output,
                                                                                         d_count, count_cap); count_launch();
    return cudaGetLastError();
}

size_t mt19937_padded(size_t count) { return (count + 2 * MT_STEP - 1) / (2 * MT_STEP) * (2 * MT_STEP); }

cudaError_t mt19937_generate(uint32_t seed, uint32_t* out, size_t have, size_t need, uint32_t* ring, cudaStream_t st) {
    MtSeed s;
    s.x[0] = seed;
    for (uint32_t i = 1; i < MT_N; i++) s.x[i] = 1812433253u * (s.x[i - 1] ^ (s.x[i - 1] >> 30)) + i;
    k_mt19937<<<1, 256, 0, st>>>(s, ring, have / MT_STEP, (need - have) / MT_STEP, out); count_launch();
    return cudaGetLastError();
}

void gen_mt19937(uint32_t seed, uint64_t count, uint32_t* out) {
    std::mt19937 g(seed);
    for (uint64_t i = 0; i < count; i++) out[i] = (uint32_t)g();
}

}  // namespace nnm
