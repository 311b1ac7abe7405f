// Copies between pageable host memory and the device (hostcopy.cu).
#pragma once
#include <cstddef>
#include <cstdint>

#include <cuda_runtime.h>

namespace nnm {

struct Ctx;

struct CopyThreads;  // hostcopy.cu

// Pinned slots the copies pass through and the threads that fill and empty
// them, owned by a context: made by the first copy that uses them, freed and
// joined with the context.
struct HostStage {
    static constexpr int WORKERS = 4, SLOTS = 2;
    static constexpr size_t CHUNK = (size_t)1 << 20;
    unsigned char* block = nullptr;  // WORKERS x SLOTS x CHUNK
    cudaEvent_t done[WORKERS][SLOTS] = {};
    bool failed = false;  // no pinned memory: plain copies
    CopyThreads* threads = nullptr;
    void release();
};

struct HostPiece {
    void* host;
    const void* dev;
    size_t bytes;
};

// Pinned memory (freed with cudaFreeHost), or null where there is none: the
// callers then copy without it.
unsigned char* pinned_block(size_t bytes);
// dst[0, bytes) = src, ordered on the context's stream; src may change once
// the call returns (it waits for the copy of pinned or managed memory).
cudaError_t host_to_dev(Ctx& ctx, void* dst, const void* src, size_t bytes);
// Every piece's device bytes to its host memory, after the work on the
// context's stream; complete when the call returns.  Pieces with a null host
// pointer are skipped.
cudaError_t dev_to_host(Ctx& ctx, const HostPiece* pieces, int count);

}  // namespace nnm
