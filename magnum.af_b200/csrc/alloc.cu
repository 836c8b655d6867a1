// Device memory of DevBuf.  cudaMalloc and cudaFree of more than about 1 MB take 0.3-4 ms
// each here (mapping and unmapping), which was most of a new DemagField (7-12 ms for
// 200x120x10 cells, 2.5 of them kernels) and of a new state's first step.  Allocations of
// up to kPoolMax bytes therefore come from a memory pool of the device that keeps up to
// kPoolKeep unused bytes for the next object and gives the rest back to the driver at the
// next synchronisation; larger ones are cudaMalloc's.
//
// The pool belongs to this library (the device's default pool and its settings are left
// alone) and is used on one internal stream: an allocation is synchronised before it is
// handed out, and a buffer goes back only after the device has finished all work that may
// use it (as cudaFree waits), so the buffers may be used on any stream and from any thread.
#include <mutex>

#include "engine.hpp"

namespace mafb {

namespace {

constexpr size_t kPoolMax = 128u << 20;
constexpr unsigned long long kPoolKeep = 256ull << 20;
constexpr int kMaxOrdinals = 64;

struct DevicePool {
    cudaMemPool_t pool = nullptr;
    cudaStream_t stream = nullptr;
    bool failed = false;
};

// The device's pool, made on first use; null when there is none (the caller uses cudaMalloc).
DevicePool* device_pool() {
    static std::mutex mu;
    static DevicePool pools[kMaxOrdinals];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxOrdinals) return nullptr;
    std::lock_guard<std::mutex> lock(mu);
    DevicePool& p = pools[dev];
    if (!p.pool && !p.failed) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        unsigned long long keep = kPoolKeep;
        p.failed = cudaMemPoolCreate(&p.pool, &props) != cudaSuccess ||
                   cudaMemPoolSetAttribute(p.pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess ||
                   cudaStreamCreateWithFlags(&p.stream, cudaStreamNonBlocking) != cudaSuccess;
        if (p.failed) cudaGetLastError();
    }
    return p.failed ? nullptr : &p;
}

}  // namespace

void* dev_alloc(size_t n) {
    void* ptr = nullptr;
    if (n <= kPoolMax) {
        if (DevicePool* p = device_pool()) {
            if (cudaMallocFromPoolAsync(&ptr, n, p->pool, p->stream) == cudaSuccess &&
                cudaStreamSynchronize(p->stream) == cudaSuccess)
                return ptr;
            // no memory for the pool to grow, or a context that was reset under it
            cudaGetLastError();
            ptr = nullptr;
        }
    }
    MAF_CUDA(cudaMalloc(&ptr, n));
    return ptr;
}

void dev_free(void* ptr, size_t n) {
    if (n > kPoolMax) {
        cudaFree(ptr);
        return;
    }
    int dev = 0;
    cudaPointerAttributes at = {};
    cudaGetDevice(&dev);
    if (cudaPointerGetAttributes(&at, ptr) != cudaSuccess) {
        cudaGetLastError();  // the context is gone, and the memory with it
        return;
    }
    if (at.device != dev) cudaSetDevice(at.device);
    // (a device that cannot be synchronised, as inside a capture, keeps the buffer)
    if (cudaDeviceSynchronize() == cudaSuccess) {
        DevicePool* p = device_pool();
        if (!p || cudaFreeAsync(ptr, p->stream) != cudaSuccess) {
            cudaGetLastError();
            cudaFree(ptr);  // not the pool's
        }
    } else {
        cudaGetLastError();
    }
    if (at.device != dev) cudaSetDevice(dev);
}

}  // namespace mafb
