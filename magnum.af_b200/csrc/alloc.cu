// Device memory of DevBuf.  cudaMalloc and cudaFree of more than about 1 MB take 0.3-4 ms
// each here (mapping and unmapping), which was most of a new DemagField (7-12 ms for
// 200x120x10 cells, 2.5 of them kernels) and of a new state's first step.  Allocations of
// up to kPoolMax bytes therefore come from a memory pool of the device that keeps up to
// kPoolKeep unused bytes for the next object and gives the rest back to the driver at the
// next synchronisation; larger ones are cudaMalloc's, and so are the buffers whose address
// the application gets (DevBuf::alloc_own): pool memory has neither the IPC handles nor the
// peer access of cudaMalloc memory.  Of these up to kPoolKeep bytes are kept, too, for the next
// state of the same size (300x200 cells, a new state's first step: 2.5 ms without, 0.7 with; the
// two buffers are 1.4 MB each).  dev_trim gives everything unused back.
//
// The pool belongs to this library (the device's default pool and its settings are left
// alone) and is used on one internal stream: an allocation is synchronised before it is
// handed out, and a buffer goes back only after the device has finished all work that may
// use it, so the buffers may be used on any stream and from any thread.  That wait is a
// cudaFree of a small block (which waits for all streams of the device, 5 us with the next
// block at hand), not cudaDeviceSynchronize: a thread may free while another one captures a
// graph in thread-local mode, where the latter is not allowed and spoils the capture.
#include <mutex>
#include <vector>

#include "engine.hpp"

namespace mafb {

namespace {

constexpr size_t kPoolMax = 128u << 20;
constexpr unsigned long long kPoolKeep = 256ull << 20;
constexpr int kMaxOrdinals = 64;
constexpr size_t kSmall = 64;

struct Block {
    void* p;
    size_t n;
};

struct DevicePool {
    cudaMemPool_t pool = nullptr;
    cudaStream_t stream = nullptr;
    void* anchor = nullptr;        // keeps the driver's block of small allocations (340 us to make, 280 to unmake)
    bool failed = false;
    std::mutex mu;
    std::vector<void*> pending;    // pool buffers whose device could not be waited for yet
    std::vector<Block> own;        // unused cudaMalloc'd buffers, oldest first
    size_t own_bytes = 0;
};

// The device's pool, made on first use; null when there is none (the caller uses cudaMalloc).
DevicePool* device_pool() {
    static std::mutex mu;
    static DevicePool* pools = new DevicePool[kMaxOrdinals];  // (outlives the buffers of static objects)
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
        p.failed = cudaMalloc(&p.anchor, kSmall) != cudaSuccess ||
                   cudaMemPoolCreate(&p.pool, &props) != cudaSuccess ||
                   cudaMemPoolSetAttribute(p.pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess ||
                   cudaStreamCreateWithFlags(&p.stream, cudaStreamNonBlocking) != cudaSuccess;
        if (p.failed) cudaGetLastError();
    }
    return p.failed ? nullptr : &p;
}

// Waits for all work of the device as cudaFree does; false where cudaFree is not allowed (a
// thread that is capturing itself).
bool wait_device() {
    void* w = nullptr;
    if (cudaMalloc(&w, kSmall) == cudaSuccess && cudaFree(w) == cudaSuccess) return true;
    cudaGetLastError();
    return false;
}

// Gives ptr (may be null; idle: nothing uses it any more) and the pending buffers back to the
// pool, or keeps them pending.
void give_back(DevicePool& p, void* ptr, bool idle) {
    if (ptr && idle) {
        cudaFreeAsync(ptr, p.stream);
        return;
    }
    std::vector<void*> list;
    {
        std::lock_guard<std::mutex> lock(p.mu);
        list.swap(p.pending);
    }
    if (ptr) list.push_back(ptr);
    if (list.empty()) return;
    if (wait_device()) {
        for (void* q : list) cudaFreeAsync(q, p.stream);
        return;
    }
    std::lock_guard<std::mutex> lock(p.mu);
    p.pending.insert(p.pending.end(), list.begin(), list.end());
}

void* take_own(DevicePool& p, size_t n) {
    std::lock_guard<std::mutex> lock(p.mu);
    for (auto b = p.own.begin(); b != p.own.end(); ++b)
        if (b->n == n) {
            void* q = b->p;
            p.own_bytes -= n;
            p.own.erase(b);
            return q;
        }
    return nullptr;
}

// Keeps an unused buffer and frees the oldest ones beyond `keep` bytes.
void keep_own(DevicePool& p, Block b, size_t keep) {
    std::vector<Block> out;
    {
        std::lock_guard<std::mutex> lock(p.mu);
        if (b.p) {
            p.own.push_back(b);
            p.own_bytes += b.n;
        }
        while (p.own_bytes > keep) {
            out.push_back(p.own.front());
            p.own_bytes -= p.own.front().n;
            p.own.erase(p.own.begin());
        }
    }
    for (const Block& o : out) cudaFree(o.p);
}

void trim(DevicePool& p) {
    give_back(p, nullptr, false);
    keep_own(p, Block{nullptr, 0}, 0);
    cudaStreamSynchronize(p.stream);
    cudaMemPoolTrimTo(p.pool, 0);
    cudaGetLastError();
}

}  // namespace

void dev_trim() {
    if (DevicePool* p = device_pool()) trim(*p);
}

void* dev_alloc(size_t n, bool own, bool* pooled) {
    void* ptr = nullptr;
    DevicePool* p = device_pool();
    *pooled = false;
    if (p && !own && n <= kPoolMax) {
        if (cudaMallocFromPoolAsync(&ptr, n, p->pool, p->stream) == cudaSuccess) {
            if (cudaStreamSynchronize(p->stream) == cudaSuccess) {
                *pooled = true;
                return ptr;
            }
            cudaFreeAsync(ptr, p->stream);
        }
        // no memory for the pool to grow, or a context that was reset under it
        cudaGetLastError();
        ptr = nullptr;
    }
    if (p && own && n <= kPoolMax && (ptr = take_own(*p, n))) return ptr;
    cudaError_t e = cudaMalloc(&ptr, n);
    if (e == cudaErrorMemoryAllocation && p) {  // what is kept unused may be enough
        cudaGetLastError();
        trim(*p);
        e = cudaMalloc(&ptr, n);
    }
    if (e != cudaSuccess) cudaGetLastError();
    MAF_CUDA(e);
    return ptr;
}

void dev_free(void* ptr, size_t n, bool pooled, bool idle) {
    if (!pooled && n > kPoolMax) {
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
    DevicePool* p = device_pool();
    if (pooled && p)
        give_back(*p, ptr, idle);
    else if (p && (idle || wait_device()))
        keep_own(*p, Block{ptr, n}, kPoolKeep);
    else
        cudaFree(ptr);
    if (at.device != dev) cudaSetDevice(dev);
}

void release_all(const std::vector<DevBuf*>& bufs) {
    const DevBuf* any = nullptr;
    for (const DevBuf* b : bufs)
        if (b->p) any = b;
    if (!any) return;
    int dev = 0;
    cudaPointerAttributes at = {};
    cudaGetDevice(&dev);
    if (cudaPointerGetAttributes(&at, any->p) != cudaSuccess) {
        cudaGetLastError();
        at.device = dev;
    }
    if (at.device != dev) cudaSetDevice(at.device);
    const bool idle = wait_device();
    if (at.device != dev) cudaSetDevice(dev);
    for (DevBuf* b : bufs) b->release(idle);
}

}  // namespace mafb
