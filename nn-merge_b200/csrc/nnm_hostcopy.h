// Copies between pageable host memory and the device (hostcopy.cu).
#pragma once
#include <sys/types.h>

#include <cstddef>
#include <cstdint>

#include <cuda_runtime.h>

namespace nnm {

struct Ctx;

struct CopyThreads;  // hostcopy.cu

// Page-locked memory of one process: mapped here and registered (8 MB on huge
// pages: 0.6 ms and 0.15 to give back; cudaMallocHost 1.5 and 0.5, on other hosts
// 6 and 1), not inherited by a forked child.
struct PinnedBlock {
    unsigned char* p = nullptr;
    size_t bytes = 0;
    pid_t owner = 0;
    bool make(size_t n);  // false where there is none: the callers then copy without it
    bool here() const;    // the calling process made it
    void release();
};

// Pinned slots the copies pass through and the threads that fill and empty
// them, owned by a context: made by the first copy that uses them (the first
// worker's; the others' by the first copy that is shared), freed and joined
// with the context.
struct HostStage {
    static constexpr int WORKERS = 4, SLOTS = 2;
    static constexpr size_t CHUNK = (size_t)1 << 20;
    PinnedBlock first, others;  // SLOTS chunks of worker 0; of the other workers
    cudaEvent_t done[WORKERS][SLOTS] = {};
    bool failed = false;  // no pinned memory: plain copies
    CopyThreads* threads = nullptr;
    unsigned char* slot(int w, int i) const {
        return w == 0 ? first.p + (size_t)i * CHUNK : others.p + ((size_t)(w - 1) * SLOTS + i) * CHUNK;
    }
    void release();
};

struct HostPiece {
    void* host;
    const void* dev;
    size_t bytes;
};

// dst[0, bytes) = src, ordered on the context's stream; src may change once
// the call returns (it waits for the copy of pinned or managed memory).
cudaError_t host_to_dev(Ctx& ctx, void* dst, const void* src, size_t bytes);
// Every piece's device bytes to its host memory, after the work on the
// context's stream; complete when the call returns.  Pieces with a null host
// pointer are skipped.
cudaError_t dev_to_host(Ctx& ctx, const HostPiece* pieces, int count);

}  // namespace nnm
