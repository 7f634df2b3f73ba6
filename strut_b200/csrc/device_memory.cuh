// Device memory of the library's objects and shared memory of its kernels (included once, by strut_cuda.cu).
//
// Creating and destroying an analysis used to make some seventy cudaMalloc / cudaFree calls, each of
// which maps or unmaps memory and can wait for the whole device: 4 to 40 ms a handle, with single
// calls of up to 400 ms.  Objects now take their arrays from an arena of a few blocks, and the
// blocks come from one stream-ordered pool per device, which keeps at most kPoolKeep bytes between
// objects (the rest goes back to the device as blocks are freed; everything does when an allocation
// fails, and at the end of the process).  Pools are safe to use from several threads and streams: a
// block freed on one stream is handed out again only once that stream has passed the free.
#pragma once

#include <algorithm>
#include <mutex>
#include <vector>

namespace {

constexpr int kPoolDevices = 64;
constexpr unsigned long long kPoolKeep = 1ull << 30;
constexpr size_t kArenaBlock = 16u << 20;  // arrays up to a quarter of it share blocks
std::mutex g_pool_mu;
cudaMemPool_t g_pool[kPoolDevices];

int pool_of_device(cudaMemPool_t* out) {
    int dev = 0;
    CK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kPoolDevices) return fail(STRUT_UNSUPPORTED, "device index too large");
    std::lock_guard<std::mutex> lock(g_pool_mu);
    if (!g_pool[dev]) {
        cudaMemPoolProps pp;
        std::memset(&pp, 0, sizeof(pp));
        pp.allocType = cudaMemAllocationTypePinned;
        pp.location.type = cudaMemLocationTypeDevice;
        pp.location.id = dev;
        cudaMemPool_t p = nullptr;
        CK(cudaMemPoolCreate(&p, &pp));
        unsigned long long keep = kPoolKeep;
        CK(cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep));
        g_pool[dev] = p;
    }
    *out = g_pool[dev];
    return STRUT_OK;
}

// A block of the current device's pool, usable on stream s (elsewhere once s has passed here).
int pool_alloc(void** p, size_t bytes, cudaStream_t s) {
    cudaMemPool_t pool;
    const int rc = pool_of_device(&pool);
    if (rc != STRUT_OK) return rc;
    bytes = std::max<size_t>(bytes, 16);
    if (cudaMallocFromPoolAsync(p, bytes, pool, s) == cudaSuccess) return STRUT_OK;
    cudaGetLastError();
    CK(cudaDeviceSynchronize());
    CK(cudaMemPoolTrimTo(pool, 0));
    CK(cudaMallocFromPoolAsync(p, bytes, pool, s));
    return STRUT_OK;
}

// Zeroed device arrays of one object, all on one stream; given back together.
struct Arena {
    cudaStream_t s = nullptr;
    std::vector<void*> blocks;
    char* cur = nullptr;
    size_t left = 0;
    int dev = 0;  // device of the blocks
    int take(void** p, size_t bytes) {
        bytes = (std::max<size_t>(bytes, 1) + 255) & ~(size_t)255;
        if (bytes > left) {
            const bool own = bytes > kArenaBlock / 4;
            const size_t size = own ? bytes : kArenaBlock;
            void* b = nullptr;
            const int rc = pool_alloc(&b, size, s);
            if (rc != STRUT_OK) return rc;
            blocks.push_back(b);
            CK(cudaGetDevice(&dev));
            CK(cudaMemsetAsync(b, 0, size, s));
            if (own) {
                *p = b;
                return STRUT_OK;
            }
            cur = (char*)b;
            left = size;
        }
        *p = cur;
        cur += bytes;
        left -= bytes;
        return STRUT_OK;
    }
    void release() {
        if (blocks.empty()) return;
        int here = 0;
        cudaGetDevice(&here);
        if (here != dev) cudaSetDevice(dev);
        // an object on the legacy default stream is used on streams of its callers
        if (!s) cudaDeviceSynchronize();
        for (void* b : blocks) cudaFreeAsync(b, s);
        if (here != dev) cudaSetDevice(here);
        blocks.clear();
        cur = nullptr;
        left = 0;
    }
};

// An array of the arena with the contents of h (the host copy is free again on return).
template <typename T>
int upload(T** dptr, const std::vector<T>& h, Arena& a) {
    const int rc = a.take((void**)dptr, h.size() * sizeof(T));
    if (rc != STRUT_OK) return rc;
    if (!h.empty()) CK(cudaMemcpyAsync(*dptr, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice, a.s));
    return STRUT_OK;
}

template <typename T>
int dzeros(T** dptr, size_t n, Arena& a) {
    return a.take((void**)dptr, n * sizeof(T));
}

// Lets a kernel take that much dynamic shared memory.  The limit belongs to the function, not to a handle, so
// it is only ever raised: set to each handle's need, it was lowered by a smaller handle and a larger
// one's next launch or graph was refused.
std::mutex g_smem_mu;
int raise_shared_memory(const void* kernel, size_t bytes) {
    std::lock_guard<std::mutex> lock(g_smem_mu);
    cudaFuncAttributes fa;
    CK(cudaFuncGetAttributes(&fa, kernel));
    if ((size_t)fa.maxDynamicSharedSizeBytes < bytes)
        CK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    return STRUT_OK;
}

}  // namespace
