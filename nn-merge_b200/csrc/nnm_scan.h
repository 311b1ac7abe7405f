#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

namespace nnm {
// One scan: out[i] = in[0] + ... + in[i-1] for i in [0, n]; out has n+1
// entries and out[n] is the total, also written to *total when non-null.
// With in2 the i-th input is max(in[i] - 1, 0) + max(in2[i] - 1, 0) instead
// (the draws that shuffling two lists of those lengths takes).  With over, a
// total above cap sets `bit` there.
struct ScanJob {
    const uint32_t *in, *in2;
    uint64_t *out, *total;
    unsigned int* over;
    uint64_t cap;
    unsigned int bit;
};
struct ScanJobs {
    static constexpr int MAX = 3;
    ScanJob j[MAX];
};
// The first `count` jobs, all over n inputs.
cudaError_t exclusive_scans(const ScanJobs& jobs, int count, size_t n, uint64_t* temp, cudaStream_t st);
// Scratch size (in u64 elements) that the scans need for n inputs.
size_t scan_temp_elems(size_t n);
// One plain scan.
cudaError_t exclusive_scan(const uint32_t* in, uint64_t* out, size_t n, uint64_t* temp, cudaStream_t st);
}  // namespace nnm
