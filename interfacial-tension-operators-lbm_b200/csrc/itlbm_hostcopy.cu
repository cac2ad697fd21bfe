// itlbm_hostcopy.cu -- device arrays to the caller's pageable host memory.
//
// A copy to pageable memory goes through the driver's own staging, one thread that copies and, for fresh
// memory, takes the page faults: on the B200 hosts 4.6 GB/s (36 ms for the five fields of a 2048 x 2048
// box, a quarter of a 500-step interval's time), and every small array costs a synchronous copy of its
// own (five fields of a 40 x 40 box: 90 us).  Here the data comes through pinned memory: what fits it in
// one copy and one wait, larger data in chunks that several threads copy out (and fault in) while the
// next ones arrive: 2048 x 2048 in 11 ms, 40 x 40 in 37 us.
#include "itlbm_internal.h"

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstring>
#include <exception>
#include <mutex>
#include <new>
#include <thread>

namespace itlbm {

namespace {

constexpr int SLOTS = 8;      // chunks in flight
constexpr int WORKERS = 8;
// Pinned memory is dear to allocate, and a program that reads each case once pays for it each time: 1 MB is had from
// what the driver holds, 4 MB take 2 to 5 ms, 16 MB 11 ms.  So small reads take 1 MB, and what large ones take
// grows with what they save: the first read of five fields of 1024 x 768 takes 4 to 7 ms (plain 8.5, with 16 MB 10
// to 18), further ones 1.6; of 2048 x 2048 25 and 11 ms (plain 37; with 4 MB 18 and 13).
constexpr size_t SMALL = (size_t)1 << 20;  // up to this in one copy, by the calling thread
constexpr size_t HUGE_READ = (size_t)64 << 20, MEDIUM_STAGE = (size_t)4 << 20, HUGE_STAGE = (size_t)16 << 20;
// From this on in chunks.  Between the two the plain copies: their arrays still come from the host
// allocator's own pages, and the threads cost more than they save (five fields of 512 x 512, 10.5 MB:
// 0.69 ms plain, 1.0 ms in chunks; of 1024 x 768, 31 MB: 8.5 and 2.2 ms).
constexpr size_t LARGE = (size_t)16 << 20;

// The pinned memory, shared by all cases and batches and used by one call at a time (a second call
// meanwhile takes the plain copy); it grows to what calls need, at most 16 MB, and is freed with the last of them.
struct Stage {
    std::mutex lock;
    char *buf = nullptr;
    size_t cap = 0;
};
Stage g_stage;
std::mutex g_refs_lock;
int g_refs = 0;

bool reserve(size_t bytes) {
    if (g_stage.cap >= bytes) return true;
    if (g_stage.buf) cudaFreeHost(g_stage.buf);
    g_stage.buf = nullptr;
    g_stage.cap = 0;
    if (cudaHostAlloc((void **)&g_stage.buf, bytes, cudaHostAllocPortable) != cudaSuccess) {
        cudaGetLastError();
        g_stage.buf = nullptr;
        return false;
    }
    g_stage.cap = bytes;
    return true;
}

cudaError_t fetch_plain(double *const *dst, int n, size_t each, const double *src, cudaStream_t st) {
    cudaError_t e = cudaSuccess;
    for (int k = 0; k < n && e == cudaSuccess; k++)
        if (dst[k]) e = cudaMemcpyAsync(dst[k], src + k * each, sizeof(double) * each, cudaMemcpyDeviceToHost, st);
    const cudaError_t s = cudaStreamSynchronize(st);
    return e == cudaSuccess ? s : e;
}

cudaError_t fetch_small(double *const *dst, int n, size_t each, const double *src, cudaStream_t st) {
    const size_t bytes = sizeof(double) * each;
    cudaError_t e = cudaMemcpyAsync(g_stage.buf, src, bytes * n, cudaMemcpyDeviceToHost, st);
    const cudaError_t s = cudaStreamSynchronize(st);
    if (e == cudaSuccess) e = s;
    for (int k = 0; k < n && e == cudaSuccess; k++)
        if (dst[k]) std::memcpy(dst[k], g_stage.buf + k * bytes, bytes);
    return e;
}

struct Chunk {
    char *dst;
    const char *src;
    size_t bytes;
};

// Chunk c comes into slot c mod SLOTS once the chunk before it there is copied out; the workers take the
// chunks in order.
cudaError_t fetch_large(const std::vector<Chunk> &chunks, cudaStream_t st) {
    const size_t n = chunks.size(), slot = g_stage.cap / SLOTS;
    std::mutex m;
    std::condition_variable cv;
    size_t issued = 0, next = 0;
    std::vector<char> done(n, 0);
    std::vector<std::thread> pool;
    pool.reserve(WORKERS);
    cudaEvent_t ev[SLOTS] = {};
    cudaError_t e = cudaSuccess;
    for (auto &v : ev)
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&v, cudaEventDisableTiming);
    cudaError_t worker_error = cudaSuccess;
    bool stop = false;
    int device = 0;
    cudaGetDevice(&device);
    auto work = [&]() {
        cudaSetDevice(device);
        std::unique_lock<std::mutex> g(m);
        for (;;) {
            const size_t c = next;
            if (c >= n) return;
            next++;
            cv.wait(g, [&] { return issued > c || stop; });
            if (issued <= c) return;
            g.unlock();
            const cudaError_t w = cudaEventSynchronize(ev[c % SLOTS]);
            if (w == cudaSuccess) std::memcpy(chunks[c].dst, g_stage.buf + (c % SLOTS) * slot, chunks[c].bytes);
            g.lock();
            if (w != cudaSuccess) worker_error = w;
            done[c] = 1;
            cv.notify_all();
        }
    };
    if (e == cudaSuccess) {
        const size_t want = std::min<size_t>({n, (size_t)WORKERS, std::max(1u, std::thread::hardware_concurrency())});
        try {
            while (pool.size() < want) pool.emplace_back(work);
        } catch (const std::exception &) {  // no thread or no memory to be had: fewer threads
        }
        if (pool.empty()) {
            for (auto &v : ev)
                if (v) cudaEventDestroy(v);
            return cudaErrorNotReady;  // the caller takes the plain copy
        }
    }
    for (size_t c = 0; c < n && e == cudaSuccess; c++) {
        {
            std::unique_lock<std::mutex> g(m);
            if (c >= SLOTS) cv.wait(g, [&] { return done[c - SLOTS] != 0; });
        }
        e = cudaMemcpyAsync(g_stage.buf + (c % SLOTS) * slot, chunks[c].src, chunks[c].bytes, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaEventRecord(ev[c % SLOTS], st);
        if (e != cudaSuccess) break;
        std::lock_guard<std::mutex> g(m);
        issued = c + 1;
        cv.notify_all();
    }
    {
        std::lock_guard<std::mutex> g(m);
        stop = true;
        cv.notify_all();
    }
    for (auto &t : pool) t.join();
    const cudaError_t s = cudaStreamSynchronize(st);
    for (auto &v : ev)
        if (v) cudaEventDestroy(v);
    return e != cudaSuccess ? e : (worker_error != cudaSuccess ? worker_error : s);
}

}  // namespace

void host_stage_ref() {
    std::lock_guard<std::mutex> g(g_refs_lock);
    g_refs++;
}

void host_stage_unref() {
    std::lock_guard<std::mutex> g(g_refs_lock);
    if (--g_refs > 0) return;
    std::lock_guard<std::mutex> s(g_stage.lock);
    if (g_stage.buf) cudaFreeHost(g_stage.buf);
    g_stage.buf = nullptr;
    g_stage.cap = 0;
}

cudaError_t fetch_arrays(double *const *dst, int n, size_t each, const double *src, cudaStream_t st) {
    size_t total = 0;
    for (int k = 0; k < n; k++) total += dst[k] ? sizeof(double) * each : 0;
    if (total == 0) return cudaStreamSynchronize(st);
    const size_t whole = sizeof(double) * each * n;
    std::unique_lock<std::mutex> g(g_stage.lock, std::try_to_lock);
    if (!g.owns_lock()) return fetch_plain(dst, n, each, src, st);
    if (whole <= SMALL) {
        if (!reserve(SMALL)) return fetch_plain(dst, n, each, src, st);
        return fetch_small(dst, n, each, src, st);
    }
    if (total < LARGE || !reserve(total < HUGE_READ ? MEDIUM_STAGE : HUGE_STAGE)) return fetch_plain(dst, n, each, src, st);
    const size_t most = g_stage.cap / SLOTS;
    cudaError_t e = cudaErrorNotReady;
    try {
        std::vector<Chunk> chunks;
        for (int k = 0; k < n; k++)
            for (size_t at = 0; dst[k] && at < sizeof(double) * each; at += most)
                chunks.push_back(Chunk{(char *)dst[k] + at, (const char *)(src + k * each) + at,
                                       std::min(most, sizeof(double) * each - at)});
        e = fetch_large(chunks, st);
    } catch (const std::bad_alloc &) {  // before any copy began
    }
    return e == cudaErrorNotReady ? fetch_plain(dst, n, each, src, st) : e;
}

}  // namespace itlbm
