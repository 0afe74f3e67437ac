// Runs csrc/host_copy.h on the CPU, against a stand-in for the few CUDA calls it makes:
// copies are memcpy, events nothing.  Prints the most threads the process had during a
// call (main included) and fails on a wrong byte.
#include <dirent.h>

#include <cstdio>
#include <cstdlib>
#include <vector>

#include "host_copy.h"

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

int main() {
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
