// hostcopy.cu over a stand-in for the CUDA runtime: copies wait in a queue
// until an event or the stream is waited for (as a device's DMA may), and a
// chosen call fails once.  Prints one line per check; exit status 1 on a
// failed one.
#include <math.h>
#include <signal.h>
#include <sys/wait.h>
#include <unistd.h>

#include <cstdio>
#include <cstdlib>
#include <deque>
#include <map>

// what the headers' device code names (none of it is called here)
float __fadd_rn(float, float), __fsub_rn(float, float), __fmul_rn(float, float), __fdiv_rn(float, float);
unsigned __umulhi(unsigned, unsigned), min(unsigned, unsigned);
int __popc(unsigned), __clz(int);

#include "../../nn-merge_b200/csrc/hostcopy.cu"

namespace {
struct Copy {
    void* dst;
    const void* src;
    size_t bytes;
};
std::mutex mu;
std::deque<Copy> queue_;
size_t done_ = 0, issued_ = 0;          // copies carried out, copies issued
std::map<cudaEvent_t, size_t> marks;    // event -> copies issued before its record
std::map<const char*, size_t> pinned;   // page-locked ranges
long calls = 0, fail_at = 0;            // the fail_at-th enqueue or record call fails
bool no_pinned = false;                 // pinned memory cannot be had
cudaError_t last_error = cudaSuccess;

void run_to(size_t upto) {
    while (done_ < upto && !queue_.empty()) {
        const Copy c = queue_.front();
        queue_.pop_front();
        std::memcpy(c.dst, c.src, c.bytes);
        done_++;
    }
}
bool is_pinned(const void* p) {
    auto it = pinned.upper_bound(static_cast<const char*>(p));
    if (it == pinned.begin()) return false;
    --it;
    return static_cast<const char*>(p) < it->first + it->second;
}
bool fails() { return ++calls == fail_at; }
}  // namespace

extern "C" {
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t bytes, cudaMemcpyKind kind, cudaStream_t) {
    std::lock_guard<std::mutex> l(mu);
    if (fails()) return cudaErrorUnknown;
    queue_.push_back({dst, src, bytes});
    issued_++;
    // pageable host memory is staged (in) or waited for (out) within the call
    if (!is_pinned(kind == cudaMemcpyHostToDevice ? src : dst)) run_to(issued_);
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) {
    std::lock_guard<std::mutex> l(mu);
    if (fails()) return cudaErrorUnknown;
    marks[e] = issued_;
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    std::lock_guard<std::mutex> l(mu);
    run_to(marks[e]);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) {
    std::lock_guard<std::mutex> l(mu);
    run_to(issued_);
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    *e = reinterpret_cast<cudaEvent_t>(std::malloc(1));
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
    std::free(e);
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t bytes) {
    std::lock_guard<std::mutex> l(mu);
    if (no_pinned) return last_error = cudaErrorMemoryAllocation;
    *p = std::malloc(bytes);
    pinned[static_cast<char*>(*p)] = bytes;
    return cudaSuccess;
}
cudaError_t cudaHostRegister(void* p, size_t bytes, unsigned) {
    std::lock_guard<std::mutex> l(mu);
    if (no_pinned) return last_error = cudaErrorMemoryAllocation;
    pinned[static_cast<char*>(p)] = bytes;
    return cudaSuccess;
}
cudaError_t cudaHostUnregister(void* p) {
    std::lock_guard<std::mutex> l(mu);
    return pinned.erase(static_cast<char*>(p)) ? cudaSuccess : cudaErrorUnknown;
}
cudaError_t cudaFreeHost(void* p) {
    std::lock_guard<std::mutex> l(mu);
    pinned.erase(static_cast<char*>(p));
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    std::lock_guard<std::mutex> l(mu);
    a->type = is_pinned(p) ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaGetLastError(void) {
    const cudaError_t e = last_error;
    last_error = cudaSuccess;
    return e;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t bytes) {
    *p = std::malloc(bytes);
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    std::free(p);
    return cudaSuccess;
}
}

namespace {
int bad = 0;
void check(bool ok, const char* what, size_t bytes, long at) {
    if (!ok) {
        bad++;
        std::printf("FAILED %s, %zu bytes, call %ld\n", what, bytes, at);
    }
}
std::vector<unsigned char> bytes_of(size_t n, unsigned seed) {
    std::vector<unsigned char> v(n);
    for (size_t i = 0; i < n; i++) v[i] = (unsigned char)((i * 2654435761u + seed) >> 13);
    return v;
}

// A failed call shows in the status, whichever it is, and nothing of the
// copy is under way when the call returns.
void errors(size_t n) {
    long total = 1;
    for (long at = 0; at < total; at++) {  // 0: none
        const auto src = bytes_of(n, 1);
        for (int out = 0; out < 2; out++) {
            nnm::Ctx ctx;
            std::vector<unsigned char> dst(n), tail(1000);
            calls = 0;
            fail_at = at;
            cudaError_t e;
            if (out) {
                const nnm::HostPiece p[] = {{dst.data(), src.data(), n}, {nullptr, src.data(), n}, {tail.data(), src.data(), 1000}};
                e = nnm::dev_to_host(ctx, p, 3);
            } else {
                e = nnm::host_to_dev(ctx, dst.data(), src.data(), n);
            }
            const bool hit = at > 0 && calls >= at;
            check((e != cudaSuccess) == hit, out ? "status of a copy out" : "status of a copy in", n, at);
            if (hit) check(queue_.empty(), "nothing under way after an error", n, at);
            total = std::max(total, calls + 1);
            cudaStreamSynchronize(nullptr);
            if (!hit) check(dst == src, "bytes", n, at);
            if (!hit && out) check(!std::memcmp(tail.data(), src.data(), 1000), "bytes of the last piece", n, at);
            ctx.stage.release();
        }
    }
    std::printf("errors: %zu bytes, %ld calls\n", n, total - 1);
}

// The source changes as soon as the call returns, while copies that still
// wait run late.
void sources(size_t n) {
    const auto src = bytes_of(n, 2);
    for (int page_locked = 0; page_locked < 2; page_locked++) {
        nnm::Ctx ctx;
        std::vector<unsigned char> dst(n);
        void* p = nullptr;
        if (page_locked) cudaMallocHost(&p, n);
        else p = std::malloc(n);
        std::memcpy(p, src.data(), n);
        calls = fail_at = 0;
        check(nnm::host_to_dev(ctx, dst.data(), p, n) == cudaSuccess, "copy in", n, 0);
        std::memset(p, 0xee, n);
        cudaStreamSynchronize(nullptr);
        check(dst == src, page_locked ? "a pinned source that changes" : "a pageable source that changes", n, 0);
        if (page_locked) cudaFreeHost(p);
        else std::free(p);
        ctx.stage.release();
    }
}

// Without pinned memory the copies still come through, and no error is left
// for a later call to report.
void without_pinned(size_t n) {
    const auto src = bytes_of(n, 3);
    nnm::Ctx ctx;
    std::vector<unsigned char> dst(n), back(n);
    calls = fail_at = 0;
    no_pinned = true;
    nnm::PinnedBlock b;
    check(!b.make(n) && !b.p && cudaGetLastError() == cudaSuccess, "no pinned block", n, 0);
    const nnm::HostPiece p{back.data(), dst.data(), n};
    check(nnm::host_to_dev(ctx, dst.data(), src.data(), n) == cudaSuccess &&
              nnm::dev_to_host(ctx, &p, 1) == cudaSuccess && back == src && cudaGetLastError() == cudaSuccess,
          "copies without pinned memory", n, 0);
    no_pinned = false;
    ctx.stage.release();
}

// A forked child has the context and none of its threads: copies and the end
// of the context return there (a child of a Python program that holds a
// context destroys it as it exits), and the parent goes on.
void forked(size_t n) {
    const auto src = bytes_of(n, 4);
    nnm::Ctx ctx;
    std::vector<unsigned char> dst(n);
    calls = fail_at = 0;
    nnm::host_to_dev(ctx, dst.data(), src.data(), n);
    cudaStreamSynchronize(nullptr);  // the child's stand-in would carry out what is queued here
    for (int copy = 0; copy < 2; copy++) {
        const pid_t pid = fork();
        if (pid == 0) {
            if (copy) nnm::host_to_dev(ctx, dst.data(), src.data(), n);
            ctx.stage.release();
            _exit(0);
        }
        int status = -1;
        bool ended = false;
        for (int i = 0; i < 500 && !ended; i++) {
            ended = waitpid(pid, &status, WNOHANG) == pid;
            if (!ended) usleep(10000);
        }
        if (!ended) {
            kill(pid, SIGKILL);
            waitpid(pid, &status, 0);
        }
        check(ended && status == 0, copy ? "a copy in a forked child" : "the end of a context in a forked child", n, 0);
    }
    std::fill(dst.begin(), dst.end(), 0);
    nnm::host_to_dev(ctx, dst.data(), src.data(), n);
    cudaStreamSynchronize(nullptr);
    check(dst == src, "a copy after a fork", n, 0);
    ctx.stage.release();
}

// Page-locking costs more than a small copy takes (8 MB: 2 to 7 ms), and a
// program may make a context for one build: a context locks a quarter for
// copies of one thread, all of it for one that several share.
void locked() {
    const auto src = bytes_of((size_t)24 << 20, 5);
    auto held = [] {
        size_t n = 0;
        for (const auto& x : pinned) n += x.second;
        return n;
    };
    nnm::Ctx ctx;
    std::vector<unsigned char> dst(src.size());
    calls = fail_at = 0;
    const nnm::HostPiece small{dst.data(), src.data(), 400000}, large{dst.data(), src.data(), (size_t)10 << 20};
    nnm::host_to_dev(ctx, dst.data(), src.data(), 1 << 20);
    check(held() == 0, "nothing locked by a small copy in", held(), 0);
    nnm::dev_to_host(ctx, &small, 1);
    check(held() <= (size_t)2 << 20, "memory locked by a small copy out", held(), 0);
    nnm::dev_to_host(ctx, &large, 1);
    nnm::host_to_dev(ctx, dst.data(), src.data(), src.size());
    check(held() <= (size_t)8 << 20, "memory locked by large copies", held(), 0);
    ctx.stage.release();
    check(held() == 0, "memory locked after the context", held(), 0);
}
}  // namespace

int main() {
    for (size_t n : {(size_t)1000, (size_t)(2 << 20), (size_t)(9 << 20) + 7, (size_t)(21 << 20) + 7}) errors(n);
    for (size_t n : {(size_t)1, (size_t)100000, (size_t)(20 << 20), (size_t)(21 << 20) + 7}) sources(n);
    for (size_t n : {(size_t)1000, (size_t)(21 << 20) + 7}) without_pinned(n);
    forked((size_t)(21 << 20) + 7);
    locked();
    return bad != 0;
}
