// Runs csrc/host_copy.h on the CPU, against a stand-in for the few CUDA calls it makes:
// copies are memcpy, events nothing.  Prints the most threads the process had during a
// call (main included) and fails on a wrong byte.  With an argument the same copies run while
// no memory is to be had: after `argument` more allocations operator new throws.
#include <dirent.h>

#include <cstdio>
#include <cstdlib>
#include <new>
#include <vector>

#include "host_copy.h"

static int g_left = -1;  // allocations until there is no memory, -1: no limit
void* operator new(size_t n) {
    if (g_left == 0) throw std::bad_alloc();
    if (g_left > 0) --g_left;
    return std::malloc(n);
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

static int g_most = 0;
static void countThreads() {
    int n = 0;
    if (DIR* d = opendir("/proc/self/task")) {
        while (dirent* e = readdir(d)) n += e->d_name[0] != '.';
        closedir(d);
    }
    if (n > g_most) g_most = n;
}

extern "C" {
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    countThreads();
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) { return (*p = std::malloc(n)) ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)1; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
}

static int withoutMemory(int allocations) {
    const size_t bytes = (size_t)3 * (8 << 20) + 5, large = vfem::kDirectMax + 4097;
    std::vector<unsigned char> a(bytes, 7), b(bytes), c(large, 1), d(large);
    vfem::PinnedRing ring;
    if (vfem::hostCopyThreads() < 1) return 1;
    g_left = allocations;
    {
        vfem::PopulateTask pages(b.data(), bytes);
    }
    g_left = allocations;
    const cudaError_t in = vfem::copyToDevice(ring, d.data(), c.data(), large, 0);
    g_left = allocations;
    const cudaError_t out = vfem::copyToHost(ring, c.data(), d.data(), large, 0);
    g_left = -1;
    // no memory for a thread: the caller's does the work; none for the transfer: an error, no
    // exception (copyToHost has used up its few on mapping the pages)
    const bool got = allocations > 0 ? in == cudaSuccess && d[large - 1] == 1 : in == cudaErrorMemoryAllocation;
    return got && (out == cudaErrorMemoryAllocation || (out == cudaSuccess && c == d)) ? 0 : 1;
}

int main(int argc, char** argv) {
    if (argc > 1) return withoutMemory(std::atoi(argv[1]));
    vfem::PinnedRing ring;
    const size_t chunk = (size_t)8 << 20;
    for (size_t bytes : {(size_t)1, chunk - 3, chunk, 3 * chunk + 5, 9 * chunk + 1}) {
        std::vector<unsigned char> a(bytes), b(bytes), c(bytes);
        for (size_t i = 0; i < bytes; ++i) a[i] = (unsigned char)(i * 2654435761u >> 13);
        if (ring.toDevice(b.data(), a.data(), bytes, 0) || ring.toHost(c.data(), b.data(), bytes, 0) || a != b || a != c) {
            std::printf("wrong copy of %zu bytes\n", bytes);
            return 1;
        }
        vfem::PopulateTask pages(c.data(), bytes);
        countThreads();
        pages.wait();
        if (a != c) return 1;  // mapping changes no contents
    }
    std::printf("%d\n", g_most);
    return 0;
}
