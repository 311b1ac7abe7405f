// Copies between pageable host memory and the device.  The driver stages such
// a copy through its own pinned buffer with one thread (10 GB/s in, 5 GB/s
// out into memory touched for the first time: 5.2 + 3.5 ms of a 100,000-row
// S-Merge of 24 ms); here up to four threads share it, each claiming chunks
// and passing them through two pinned slots of its own, so that memcpy, page
// faults and DMA overlap: 51 MB in takes 1.8 ms.  Pinned (or managed) host
// memory and copies in below SHARED_IN take the plain copy; copies out below
// SHARED_OUT pass through the slots on the calling thread, with one wait for
// all pieces.  The threads stay with the context: starting three for each copy
// cost 0.4 ms.
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstring>
#include <functional>
#include <mutex>
#include <new>
#include <system_error>
#include <thread>
#include <vector>

#include "nnm_engine.h"
#include "nnm_hostcopy.h"

namespace nnm {

// Threads that run one job at a time, job(1 ..) on them and job(0) on the
// caller.  One caller at a time (a context is not thread-safe).
struct CopyThreads {
    std::mutex m;
    std::condition_variable wake, idle;
    const std::function<void(int)>* job = nullptr;
    uint64_t round = 0;
    int busy = 0;
    bool stop = false;
    std::vector<std::thread> t;

    // Fewer than asked when the system has no more threads.
    CopyThreads(int device, int n) {
        try {
            t.reserve((size_t)n);
            for (int i = 0; i < n; i++) t.emplace_back([this, device, i] { loop(device, i + 1); });
        } catch (const std::system_error&) {
        } catch (const std::bad_alloc&) {
        }
    }
    ~CopyThreads() {
        {
            std::lock_guard<std::mutex> l(m);
            stop = true;
        }
        wake.notify_all();
        for (auto& x : t) x.join();
    }
    void loop(int device, int id) {
        cudaSetDevice(device);
        uint64_t seen = 0;
        for (;;) {
            std::unique_lock<std::mutex> l(m);
            wake.wait(l, [&] { return stop || round != seen; });
            if (stop) return;
            seen = round;
            const std::function<void(int)>* f = job;
            l.unlock();
            (*f)(id);
            l.lock();
            if (--busy == 0) idle.notify_one();
        }
    }
    void run(const std::function<void(int)>& f) {
        {
            std::lock_guard<std::mutex> l(m);
            job = &f;
            busy = (int)t.size();
            round++;
        }
        wake.notify_all();
        f(0);
        std::unique_lock<std::mutex> l(m);
        idle.wait(l, [&] { return busy == 0; });
    }
};

namespace {

// below: waking the threads costs what they save.  In, whole calls, plain and
// shared: 10 MB 0.61 and 0.69 to 1.00 ms, 16 MB 0.94 and 1.06 to 1.11, 20 MB 1.17
// to 1.31 and 1.22 to 1.24, 28 MB 1.58 and 1.43 to 1.49, 51 MB 2.9 and 2.1 (a host
// whose driver stages 17 GB/s; at 10 GB/s the copies alone: 5 MB 0.45 and 0.65,
// 12 MB 1.05 and 0.7, 51 MB 5.0 and 1.8).  Out, where new pages are touched, 10
// MB: 3.8 and 1.9.
constexpr size_t SHARED_IN = (size_t)20 << 20, SHARED_OUT = (size_t)8 << 20;

bool pageable(const void* p) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

// The slots of the first worker.  A forked child has a stage without its
// threads and without its memory.
bool stage_ready(HostStage& s) {
    if (s.first.p) return s.first.here();
    if (s.failed) return false;
    bool ok = s.first.make(HostStage::SLOTS * HostStage::CHUNK);
    if (ok)
        for (auto& w : s.done)
            for (auto& e : w) ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
    if (!ok) {
        cudaGetLastError();
        s.release();
        s.failed = true;
    }
    return ok;
}

// Runs work(w) on the caller (w = 0) and, with several workers, on the
// context's copy threads; the workers claim their chunks, so none is left out
// where there are fewer threads.
void run_workers(Ctx& ctx, int workers, const std::function<void(int)>& work) {
    if (workers <= 1) {
        work(0);
        return;
    }
    if (!ctx.stage.threads) ctx.stage.threads = new (std::nothrow) CopyThreads(ctx.device, workers - 1);
    if (ctx.stage.threads) ctx.stage.threads->run(work);
    else work(0);
}

int workers_for(HostStage& s, bool shared) {
    const unsigned hw = std::thread::hardware_concurrency();
    const int most = (int)std::min<unsigned>(HostStage::WORKERS, std::max(1u, hw / 2));
    if (!shared || most == 1) return 1;
    if (!s.others.p && !s.others.make((HostStage::WORKERS - 1) * HostStage::SLOTS * HostStage::CHUNK)) return 1;
    return most;
}

// Chunks small enough that every worker gets a few.
size_t chunk_for(size_t bytes, int workers) {
    const size_t c = (bytes / ((size_t)workers * 4) + 65535) & ~(size_t)65535;
    return std::min(std::max(c, (size_t)128 << 10), HostStage::CHUNK);
}

// A copy's status once its failure is known: copies already under way end
// first, so that neither the slots (whose event may be the call that failed)
// nor the caller's memory are still in use.
cudaError_t settled(Ctx& ctx, cudaError_t e) {
    if (e != cudaSuccess) cudaStreamSynchronize(ctx.stream);
    return e;
}

}  // namespace

bool PinnedBlock::make(size_t n) {
    constexpr size_t HUGE = (size_t)2 << 20;
    n = (n + 4095) & ~(size_t)4095;
    const size_t align = n >= HUGE ? HUGE : 4096;
    void* raw = mmap(nullptr, n + align, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    if (raw == MAP_FAILED) return false;
    unsigned char* const r = static_cast<unsigned char*>(raw);
    unsigned char* const b = r + (align - reinterpret_cast<uintptr_t>(r) % align) % align;
    if (b > r) munmap(r, b - r);
    if (b + n < r + n + align) munmap(b + n, r + align - b);
    if (align == HUGE) madvise(b, n, MADV_HUGEPAGE);
    // a fork would leave the pages shared, and a write move this process's
    // away from those that the device knows
    madvise(b, n, MADV_DONTFORK);
    if (cudaHostRegister(b, n, cudaHostRegisterDefault) != cudaSuccess) {
        cudaGetLastError();
        munmap(b, n);
        return false;
    }
    p = b;
    bytes = n;
    owner = getpid();
    return true;
}

bool PinnedBlock::here() const { return p && owner == getpid(); }

void PinnedBlock::release() {
    if (here()) {
        cudaHostUnregister(p);
        munmap(p, bytes);
    }
    p = nullptr;
}

void HostStage::release() {
    // In a forked child there are no threads to join, and destroying the
    // condition that they wait on would wait for good.
    if (threads && first.here()) delete threads;
    threads = nullptr;
    for (auto& w : done)
        for (auto& e : w) {
            if (e) cudaEventDestroy(e);
            e = nullptr;
        }
    others.release();
    first.release();
}

cudaError_t host_to_dev(Ctx& ctx, void* dst, const void* src, size_t bytes) {
    HostStage& s = ctx.stage;
    const bool paged = pageable(src);
    if (bytes < SHARED_IN || !paged || !stage_ready(s)) {
        const cudaError_t e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, ctx.stream);
        // pageable memory is staged within the call; pinned and managed memory
        // is read while the copy runs
        return e == cudaSuccess && !paged ? cudaStreamSynchronize(ctx.stream) : e;
    }
    const int workers = workers_for(s, true);
    const size_t chunk = chunk_for(bytes, workers), chunks = (bytes + chunk - 1) / chunk;
    std::atomic<size_t> next{0};
    std::atomic<int> err{cudaSuccess};
    run_workers(ctx, workers, [&](int w) {
        cudaError_t e = cudaSuccess;
        for (int slot = 0; e == cudaSuccess; slot ^= 1) {
            const size_t c = next.fetch_add(1);
            if (c >= chunks) break;
            const size_t o = c * chunk, len = std::min(chunk, bytes - o);
            unsigned char* p = s.slot(w, slot);
            e = cudaEventSynchronize(s.done[w][slot]);  // the slot's last copy, of this call or an earlier one
            if (e != cudaSuccess) break;
            std::memcpy(p, static_cast<const unsigned char*>(src) + o, len);
            e = cudaMemcpyAsync(static_cast<unsigned char*>(dst) + o, p, len, cudaMemcpyHostToDevice, ctx.stream);
            if (e == cudaSuccess) e = cudaEventRecord(s.done[w][slot], ctx.stream);
        }
        if (e != cudaSuccess) err = e;
    });
    return settled(ctx, (cudaError_t)err.load());
}

cudaError_t dev_to_host(Ctx& ctx, const HostPiece* pieces, int count) {
    HostStage& s = ctx.stage;
    size_t total = 0;
    bool paged = true;
    for (int i = 0; i < count; i++)
        if (pieces[i].host && pieces[i].bytes) {
            total += pieces[i].bytes;
            paged = paged && pageable(pieces[i].host);
        }
    if (!paged || !stage_ready(s)) {
        for (int i = 0; i < count; i++)
            if (pieces[i].host && pieces[i].bytes) {
                const cudaError_t e = cudaMemcpyAsync(pieces[i].host, pieces[i].dev, pieces[i].bytes,
                                                      cudaMemcpyDeviceToHost, ctx.stream);
                if (e != cudaSuccess) return settled(ctx, e);
            }
        return cudaStreamSynchronize(ctx.stream);
    }
    if (total == 0) return cudaStreamSynchronize(ctx.stream);
    const int workers = workers_for(s, total >= SHARED_OUT);
    const size_t chunk = chunk_for(total, workers);
    size_t chunks = 0;
    for (int i = 0; i < count; i++)
        if (pieces[i].host) chunks += (pieces[i].bytes + chunk - 1) / chunk;
    // chunk c: its host and device addresses and length
    auto where = [&](size_t c, unsigned char*& h, const unsigned char*& d) -> size_t {
        for (int i = 0; i < count; i++) {
            if (!pieces[i].host) continue;
            const size_t n = (pieces[i].bytes + chunk - 1) / chunk;
            if (c < n) {
                h = static_cast<unsigned char*>(pieces[i].host) + c * chunk;
                d = static_cast<const unsigned char*>(pieces[i].dev) + c * chunk;
                return std::min(chunk, pieces[i].bytes - c * chunk);
            }
            c -= n;
        }
        return 0;
    };
    std::atomic<size_t> next{0};
    std::atomic<int> err{cudaSuccess};
    run_workers(ctx, workers, [&](int w) {
        cudaError_t e = cudaSuccess;
        unsigned char* host[HostStage::SLOTS] = {};
        size_t len[HostStage::SLOTS] = {};
        auto start = [&](int slot) {  // the next chunk on its way into the slot
            len[slot] = 0;
            const size_t c = next.fetch_add(1);
            if (c >= chunks || e != cudaSuccess) return;
            const unsigned char* d = nullptr;
            const size_t n = where(c, host[slot], d);
            e = cudaEventSynchronize(s.done[w][slot]);
            if (e == cudaSuccess) e = cudaMemcpyAsync(s.slot(w, slot), d, n, cudaMemcpyDeviceToHost, ctx.stream);
            if (e == cudaSuccess) e = cudaEventRecord(s.done[w][slot], ctx.stream);
            if (e == cudaSuccess) len[slot] = n;
        };
        for (int slot = 0; slot < HostStage::SLOTS; slot++) start(slot);
        for (int slot = 0; e == cudaSuccess && len[slot]; slot ^= 1) {  // ends with the first error
            e = cudaEventSynchronize(s.done[w][slot]);
            if (e != cudaSuccess) break;
            std::memcpy(host[slot], s.slot(w, slot), len[slot]);
            start(slot);
        }
        if (e != cudaSuccess) err = e;
    });
    const cudaError_t e = (cudaError_t)err.load();
    return e != cudaSuccess ? settled(ctx, e) : cudaStreamSynchronize(ctx.stream);
}

}  // namespace nnm
