// host_copy.h -- copies between the caller's arrays and the device.
//
// Grace and the GPU share page tables: a copy from or into the caller's own
// (pageable) pages runs at the C2C rate, without a pinned buffer.  Measured
// on GB300: 8 MB in 0.06 ms (one thread's copy into a pinned buffer alone: 0.27),
// 160 MB in 0.95 ms (9.0; 1.9 on 8 threads).  Two things make it slow, and have
// an answer here:
//   - pages that were never touched, as in a freshly allocated result array: the
//     GPU's writes fault them in one by one (160 MB: 7 to 19 ms).  PopulateTask
//     maps them, without changing what they hold, while the kernels run.
//   - large arrays: from about 250 MB the GPU's translations no longer stay
//     cached from call to call (377 MB: 2 to 48 ms for the same copy).  Above
//     kDirectMax copies go through PinnedRing, host threads and the DMA overlapped,
//     which takes the same time every time (377 MB: 2.9 ms in, about 6 out).
#pragma once

#include <sys/mman.h>
#include <unistd.h>

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <exception>
#include <new>
#include <thread>
#include <vector>

namespace vfem {

// Threads that host copies and page mapping may use: 8, or VFEM_HOST_COPY_THREADS (read once),
// and no more than the machine has.
inline size_t hostCopyThreads() {
    static const size_t n = [] {
        const char* v = std::getenv("VFEM_HOST_COPY_THREADS");
        char* end = nullptr;
        const long long x = v && *v ? std::strtoll(v, &end, 10) : 8;
        const long long want = end && *end ? 8 : std::max(1ll, x);
        return (size_t)std::min<long long>(want, std::max(1u, std::thread::hardware_concurrency()));
    }();
    return n;
}

// Maps [p, p + bytes) writable (MADV_POPULATE_WRITE, Linux 5.14).  A kernel without it
// leaves the pages to fault on use.
inline void populatePages(void* p, size_t bytes) {
    static const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE);
    const uintptr_t a = (uintptr_t)p & ~(page - 1), e = (uintptr_t)p + bytes;
    constexpr int kPopulateWrite = 23;
    if (bytes) (void)madvise((void*)a, e - a, kPopulateWrite);
}

// The same on up to hostCopyThreads() threads of 4 MB or more, done when wait() or the destructor returns.
class PopulateTask {
   public:
    PopulateTask(void* p, size_t bytes) {
        constexpr size_t kSlice = (size_t)4 << 20;
        const size_t n = std::min(hostCopyThreads(), (bytes + kSlice - 1) / kSlice);
        if (n <= 1) {
            populatePages(p, bytes);
            return;
        }
        const size_t each = (bytes + n - 1) / n;
        for (size_t i = 0; i < n; ++i) {
            char* s = (char*)p + i * each;
            const size_t len = std::min(each, bytes - i * each);
            try {
                threads_.emplace_back([s, len] { populatePages(s, len); });
            } catch (const std::exception&) {
                populatePages(s, len);  // no thread (or no memory for one) to be had
            }
        }
    }
    void wait() {
        for (auto& t : threads_) t.join();
        threads_.clear();
    }
    ~PopulateTask() { wait(); }
    PopulateTask(const PopulateTask&) = delete;
    PopulateTask& operator=(const PopulateTask&) = delete;

   private:
    std::vector<std::thread> threads_;
};

constexpr size_t kDirectMax = (size_t)192 << 20;

// Pinned chunks that host threads fill (or empty) while the DMA moves others.
// Made on first use, freed with its owner; one transfer at a time.
class PinnedRing {
   public:
    ~PinnedRing() {
        for (cudaEvent_t e : ev_)
            if (e) cudaEventDestroy(e);
        if (buf_) cudaFreeHost(buf_);
    }
    // src may be reused on return; the copies are ordered on the stream.
    cudaError_t toDevice(void* dst, const void* src, size_t bytes, cudaStream_t st) {
        cudaError_t e = init();
        if (e != cudaSuccess) return e;
        const int n = chunks(bytes);
        Workers w(n, [=](int c, size_t off, size_t len) {
            std::memcpy(slot(c) + off, (const char*)src + c * kChunk + off, len);
        }, bytes);
        w.allow(std::min(n, kSlots));
        for (int c = 0; c < n; ++c) {
            w.await(c);
            if ((e = cudaMemcpyAsync((char*)dst + c * kChunk, slot(c), size(c, bytes), cudaMemcpyHostToDevice, st)) ||
                (e = cudaEventRecord(ev_[c % kSlots], st)))
                break;
            if (c > 0) {  // the previous chunk's buffer
                if ((e = cudaEventSynchronize(ev_[(c - 1) % kSlots]))) break;
                w.allow(std::min(n, c + kSlots));
            }
        }
        w.stop();
        // the buffers still in flight are the next transfer's
        for (int c = std::max(0, n - kSlots); e == cudaSuccess && c < n; ++c) e = cudaEventSynchronize(ev_[c % kSlots]);
        return e;
    }
    // dst is complete on return.
    cudaError_t toHost(void* dst, const void* src, size_t bytes, cudaStream_t st) {
        cudaError_t e = init();
        if (e != cudaSuccess) return e;
        const int n = chunks(bytes);
        Workers w(n, [=](int c, size_t off, size_t len) {
            std::memcpy((char*)dst + c * kChunk + off, slot(c) + off, len);
        }, bytes);
        auto issue = [&](int c) {
            cudaError_t r = cudaMemcpyAsync(slot(c), (const char*)src + c * kChunk, size(c, bytes),
                                            cudaMemcpyDeviceToHost, st);
            return r != cudaSuccess ? r : cudaEventRecord(ev_[c % kSlots], st);
        };
        for (int c = 0; e == cudaSuccess && c < std::min(n, kSlots); ++c) e = issue(c);
        for (int c = 0; e == cudaSuccess && c < n; ++c) {
            if ((e = cudaEventSynchronize(ev_[c % kSlots]))) break;
            w.allow(c + 1);
            if (c > 0 && c - 1 + kSlots < n) {
                w.await(c - 1);
                e = issue(c - 1 + kSlots);
            }
        }
        if (e == cudaSuccess) w.await(n - 1);
        w.stop();
        return e;
    }

   private:
    static constexpr size_t kChunk = (size_t)8 << 20;
    static constexpr int kSlots = 4;
    char* buf_ = nullptr;
    cudaEvent_t ev_[kSlots] = {};

    char* slot(int c) const { return buf_ + (c % kSlots) * kChunk; }
    static int chunks(size_t bytes) { return (int)((bytes + kChunk - 1) / kChunk); }
    static size_t size(int c, size_t bytes) { return std::min(kChunk, bytes - c * kChunk); }
    cudaError_t init() {
        cudaError_t e = cudaSuccess;
        for (cudaEvent_t& v : ev_)
            if (!v && (e = cudaEventCreateWithFlags(&v, cudaEventDisableTiming)) != cudaSuccess) return e;
        return buf_ ? cudaSuccess : cudaMallocHost((void**)&buf_, kSlots * kChunk);
    }

    // Threads that copy their slice of chunk 0, 1, ... as each is allowed.  Where no thread
    // can be had the caller's does it (await).
    template <typename Copy>
    class Workers {
       public:
        Workers(int n, Copy copy, size_t bytes) : n_(n), copy_(copy), bytes_(bytes), done_(n) {
            for (auto& d : done_) d.store(0);
            try {
                for (int t = 0; t < (int)hostCopyThreads(); ++t) threads_.emplace_back([this, t] { run(t); });
            } catch (const std::exception&) {
            }
            count_.store(threads_.empty() ? -1 : (int)threads_.size(), std::memory_order_release);
        }
        ~Workers() { stop(); }
        void allow(int c) { allowed_.store(c, std::memory_order_release); }
        void await(int c) {
            if (threads_.empty()) {
                for (; self_ <= c; ++self_) copy_(self_, 0, size(self_, bytes_));
                return;
            }
            while (done_[c].load(std::memory_order_acquire) < (int)threads_.size()) std::this_thread::yield();
        }
        void stop() {
            stop_.store(true, std::memory_order_release);
            for (auto& t : threads_) t.join();
            threads_.clear();
        }

       private:
        void run(int t) {
            int k;
            while ((k = count_.load(std::memory_order_acquire)) == 0) std::this_thread::yield();
            for (int c = 0; c < n_; ++c) {
                while (allowed_.load(std::memory_order_acquire) <= c) {
                    if (stop_.load(std::memory_order_acquire)) return;
                    std::this_thread::yield();
                }
                const size_t len = size(c, bytes_), each = ((len + k - 1) / k + 63) & ~(size_t)63;
                const size_t off = std::min(len, t * each);
                copy_(c, off, std::min(each, len - off));
                done_[c].fetch_add(1, std::memory_order_release);
            }
        }
        const int n_;
        Copy copy_;
        const size_t bytes_;
        std::vector<std::atomic<int>> done_;
        std::atomic<int> allowed_{0}, count_{0};
        std::atomic<bool> stop_{false};
        int self_ = 0;
        std::vector<std::thread> threads_;
    };
};

// The caller's array to the device, ordered on the stream.  (Neither copy throws: they are called from C entries.)
inline cudaError_t copyToDevice(PinnedRing& ring, void* dst, const void* src, size_t bytes, cudaStream_t st) {
    try {
        return bytes > kDirectMax ? ring.toDevice(dst, src, bytes, st)
                                  : cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st);
    } catch (const std::bad_alloc&) {
        return cudaErrorMemoryAllocation;
    }
}
// Results to the caller's array; complete on return.
inline cudaError_t copyToHost(PinnedRing& ring, void* dst, const void* src, size_t bytes, cudaStream_t st) {
    PopulateTask(dst, bytes).wait();  // while the kernels before it run
    cudaError_t e;
    try {
        e = bytes > kDirectMax ? ring.toHost(dst, src, bytes, st)
                               : cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st);
    } catch (const std::bad_alloc&) {
        return cudaErrorMemoryAllocation;
    }
    return e != cudaSuccess ? e : cudaStreamSynchronize(st);
}

}  // namespace vfem
