// Staged copies between pageable host memory and the device (see gt_hostcopy.h).
#include "gt_hostcopy.h"

#include <atomic>
#include <condition_variable>
#include <cstring>
#include <mutex>
#include <new>
#include <thread>
#include <vector>

namespace gt {
namespace {
constexpr size_t kPiece = 512 * 1024;      // large enough for the link, small enough that its first byte leaves early
constexpr int kSlots = 16;                 // 8 MB of page-locked memory
constexpr int kMaxWorkers = 6;
constexpr size_t kDirect = 256 * 1024;     // below this the driver's own path is as fast
constexpr int kSpin = 20000;               // looks for the next job before a worker goes to sleep: some tens of microseconds
}  // namespace

struct HostCopier::Impl {
    char *ring = nullptr;
    cudaEvent_t done[kSlots] = {};         // the copy to / from the slot's piece has finished
    bool queued[kSlots] = {};              // ... and has been recorded at least once
    std::vector<std::thread> workers;
    std::mutex mu;
    std::condition_variable cv;
    bool stop = false;
    // the current job: pieces [0, n) between host and ring; piece i uses slot i % kSlots.  A worker takes the next piece,
    // waits until it is released (to the device: its slot is free; to the host: its bytes have arrived) and copies it.
    std::atomic<uint64_t> job{0};          // job number; workers wait for it to move
    std::atomic<int> next{0}, released{0}, busy{0};
    std::atomic<uint8_t> *ready = nullptr; // per piece: copied
    size_t ready_cap = 0;
    char *host = nullptr;
    size_t bytes = 0;
    int n = 0;
    bool in = false;                       // host -> ring

    void piece(int i) {
        const size_t at = (size_t)i * kPiece, len = bytes - at < kPiece ? bytes - at : kPiece;
        char *slot = ring + (size_t)(i % kSlots) * kPiece;
        if (in) memcpy(slot, host + at, len);
        else memcpy(host + at, slot, len);
        ready[i].store(1, std::memory_order_release);
    }
    // take and copy released pieces until none is left (wait: also wait for pieces that are not released yet)
    void help(bool wait) {
        for (;;) {
            int i = next.load(std::memory_order_relaxed);
            if (i >= n) return;
            if (i >= released.load(std::memory_order_acquire)) {
                if (!wait) return;
                std::this_thread::yield();
                continue;
            }
            if (next.compare_exchange_weak(i, i + 1, std::memory_order_acq_rel)) piece(i);
        }
    }
    void worker() {
        uint64_t seen = 0;
        for (;;) {
            uint64_t j = job.load(std::memory_order_acquire);
            for (int k = 0; j == seen && k < kSpin; k++) j = job.load(std::memory_order_acquire);
            if (j == seen) {
                std::unique_lock<std::mutex> lk(mu);
                cv.wait(lk, [&] { return stop || job.load(std::memory_order_acquire) != seen; });
                if (stop) return;
                j = job.load(std::memory_order_acquire);
            }
            seen = j;
            busy.fetch_add(1, std::memory_order_acq_rel);
            if (job.load(std::memory_order_acquire) == seen && (seen & 1)) help(true);      // odd: a job is open
            busy.fetch_sub(1, std::memory_order_acq_rel);
        }
    }
    bool open(void *h, size_t b, bool to_dev) {
        const int pieces = (int)((b + kPiece - 1) / kPiece);
        if (ready_cap < (size_t)pieces) {
            delete[] ready;
            ready = new (std::nothrow) std::atomic<uint8_t>[pieces];
            ready_cap = ready ? pieces : 0;
            if (!ready) return false;
        }
        for (int i = 0; i < pieces; i++) ready[i].store(0, std::memory_order_relaxed);
        host = (char *)h;
        bytes = b;
        n = pieces;
        in = to_dev;
        next.store(0, std::memory_order_relaxed);
        released.store(0, std::memory_order_relaxed);
        {
            std::lock_guard<std::mutex> lk(mu);
            job.fetch_add(1, std::memory_order_acq_rel);      // -> odd
        }
        cv.notify_all();
        return true;
    }
    // every piece has been taken; the job's fields may change once no worker looks at them any more
    void close() {
        next.store(n, std::memory_order_release);
        released.store(n, std::memory_order_release);
        {
            std::lock_guard<std::mutex> lk(mu);
            job.fetch_add(1, std::memory_order_acq_rel);      // -> even
        }
        while (busy.load(std::memory_order_acquire) != 0) std::this_thread::yield();
    }
    ~Impl() {
        {
            std::lock_guard<std::mutex> lk(mu);
            stop = true;
        }
        cv.notify_all();
        for (std::thread &t : workers) t.join();
        for (cudaEvent_t &e : done)
            if (e) cudaEventDestroy(e);
        if (ring) cudaFreeHost(ring);
        delete[] ready;
    }
};

HostCopier::~HostCopier() { delete impl_; }

bool HostCopier::staged(const void *host, size_t bytes) {
    if (bytes < kDirect) return false;
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, host) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

cudaError_t HostCopier::start() {
    if (impl_) return cudaSuccess;
    Impl *m = new (std::nothrow) Impl();
    if (!m) return cudaErrorMemoryAllocation;
    cudaError_t ce = cudaHostAlloc((void **)&m->ring, kSlots * kPiece, cudaHostAllocDefault);
    for (int i = 0; i < kSlots && ce == cudaSuccess; i++) ce = cudaEventCreateWithFlags(&m->done[i], cudaEventDisableTiming);
    if (ce != cudaSuccess) {
        delete m;
        return ce;
    }
    const unsigned cores = std::thread::hardware_concurrency();
    int workers = cores > 2 ? (int)cores / 2 : 1;
    if (workers > kMaxWorkers) workers = kMaxWorkers;
    try {
        for (int i = 0; i < workers; i++) m->workers.emplace_back([m] { m->worker(); });
    } catch (...) {      // fewer threads, or none: the caller copies the pieces itself
    }
    impl_ = m;
    return cudaSuccess;
}

cudaError_t HostCopier::to_device(void *dst, const void *src, size_t bytes, cudaStream_t s) {
    if (!staged(src, bytes)) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s);
    cudaError_t ce = start();
    if (ce != cudaSuccess) return ce;
    Impl &m = *impl_;
    if (!m.open(const_cast<void *>(src), bytes, true)) return cudaErrorMemoryAllocation;
    int rel = 0;
    for (int i = 0; i < m.n && ce == cudaSuccess; i++) {
        // slots whose copy of an earlier piece (of this or an earlier call) has left are handed out in order
        while (rel < m.n && rel < i + kSlots) {
            const int sl = rel % kSlots;
            if (m.queued[sl]) {
                const cudaError_t q = rel == i ? cudaEventSynchronize(m.done[sl]) : cudaEventQuery(m.done[sl]);
                if (q == cudaErrorNotReady) {
                    cudaGetLastError();
                    break;
                }
                if (q != cudaSuccess) {
                    ce = q;
                    break;
                }
                m.queued[sl] = false;
            }
            m.released.store(++rel, std::memory_order_release);
        }
        if (ce != cudaSuccess) break;
        while (!m.ready[i].load(std::memory_order_acquire)) m.help(false);
        const size_t at = (size_t)i * kPiece, len = bytes - at < kPiece ? bytes - at : kPiece;
        const int sl = i % kSlots;
        ce = cudaMemcpyAsync((char *)dst + at, m.ring + (size_t)sl * kPiece, len, cudaMemcpyHostToDevice, s);
        if (ce == cudaSuccess) ce = cudaEventRecord(m.done[sl], s);
        m.queued[sl] = ce == cudaSuccess;
    }
    m.close();
    return ce;
}

cudaError_t HostCopier::to_host(void *dst, const void *src, size_t bytes, cudaStream_t s) {
    if (!staged(dst, bytes)) {
        cudaError_t ce = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, s);
        return ce == cudaSuccess ? cudaStreamSynchronize(s) : ce;
    }
    cudaError_t ce = start();
    if (ce != cudaSuccess) return ce;
    Impl &m = *impl_;
    if (!m.open(dst, bytes, false)) return cudaErrorMemoryAllocation;
    int queued = 0;
    for (int i = 0; i < m.n && ce == cudaSuccess; i++) {
        // a slot is free again once its piece has been copied out
        while (queued < m.n && queued < i + kSlots && ce == cudaSuccess) {
            if (queued >= kSlots && !m.ready[queued - kSlots].load(std::memory_order_acquire)) {
                if (queued > i) break;
                m.help(false);
                continue;
            }
            const size_t at = (size_t)queued * kPiece, len = bytes - at < kPiece ? bytes - at : kPiece;
            const int sl = queued % kSlots;
            if (m.queued[sl] && queued < kSlots) ce = cudaEventSynchronize(m.done[sl]);      // a piece of an earlier call
            if (ce == cudaSuccess) ce = cudaMemcpyAsync(m.ring + (size_t)sl * kPiece, (const char *)src + at, len, cudaMemcpyDeviceToHost, s);
            if (ce == cudaSuccess) ce = cudaEventRecord(m.done[sl], s);
            m.queued[sl] = ce == cudaSuccess;
            queued++;
        }
        if (ce == cudaSuccess) ce = cudaEventSynchronize(m.done[i % kSlots]);
        if (ce == cudaSuccess) m.released.store(i + 1, std::memory_order_release);
    }
    if (ce == cudaSuccess)
        for (int i = 0; i < m.n; i++)
            while (!m.ready[i].load(std::memory_order_acquire)) m.help(false);
    m.close();
    return ce;
}

}  // namespace gt
