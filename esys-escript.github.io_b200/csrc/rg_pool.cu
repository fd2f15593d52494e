// The library's device memory and small pinned host blocks.
//
// A matrix, its solver vectors and its coefficient record live for one operator: a program whose
// coefficients change builds them anew every step, and a cudaMalloc or cudaFree of each costs 0.7 to
// 20 ms on a shared host (a system solve of 30,000 nodes: 34 ms when the driver is quick, 288 ms when it is
// not).  Device blocks therefore come from a stream-ordered pool of the library's own, one per device,
// which keeps at most kKept bytes that nothing uses and returns what is above it to the device at the next
// synchronisation; pinned blocks of 1 KiB are kept in a list of at most kPinned.  Both are safe for
// several threads.  As with cudaFree, a block is given back only when the device has finished all work:
// the caller may still use it on a stream that the library does not know.
//
// Large blocks (kDirect) come from cudaMalloc: kernels on arrays of hundreds of MB run slower on the pool's
// memory (a batch of 12 Bricks x 8 right hand sides 344 against 322 ms), and growing the pool by gigabytes
// takes longer (creating a 256^3 grid and matrix 70 to 90 against 6 to 11 ms).  So do blocks asked for while
// the caller's stream is captured, which cudaMalloc refuses or allows by the capture's mode; the pool would
// hand out a block of the graph.
#include <mutex>
#include <unordered_set>
#include <vector>

#include "rg_internal.cuh"

namespace rg {
namespace {

constexpr uint64_t kKept = 2ull << 30;
constexpr size_t kDirect = 64ull << 20;
constexpr size_t kPinned = 32;
constexpr int kMaxDevices = 64;

std::mutex& mutex()
{
    static std::mutex mu;
    return mu;
}

// the current device's pool; nullptr when it has none (then plain cudaMalloc is used)
cudaMemPool_t pool()
{
    static cudaMemPool_t pools[kMaxDevices] = {};
    static bool tried[kMaxDevices] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
    std::lock_guard<std::mutex> lock(mutex());
    if (!tried[dev]) {
        tried[dev] = true;
        int ok = 0;
        cudaDeviceGetAttribute(&ok, cudaDevAttrMemoryPoolsSupported, dev);
        if (ok) {
            cudaMemPoolProps p = {};
            p.allocType = cudaMemAllocationTypePinned;
            p.location.type = cudaMemLocationTypeDevice;
            p.location.id = dev;
            uint64_t keep = kKept;
            if (cudaMemPoolCreate(&pools[dev], &p) != cudaSuccess ||
                cudaMemPoolSetAttribute(pools[dev], cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) {
                cudaGetLastError();
                pools[dev] = nullptr;
            }
        }
    }
    return pools[dev];
}

// the blocks that came from cudaMalloc although there is a pool
std::unordered_set<void*>& direct()
{
    static std::unordered_set<void*> set;
    return set;
}

bool capturing()
{
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream(), &st) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    return st != cudaStreamCaptureStatusNone;
}

std::vector<void*>& pinned()
{
    static std::vector<void*> list;
    return list;
}

}  // namespace

cudaError_t dev_malloc(void** p, size_t bytes)
{
    *p = nullptr;
    cudaMemPool_t mp = pool();
    if (!mp) return cudaMalloc(p, bytes ? bytes : 1);
    if (bytes >= kDirect || capturing()) {
        cudaError_t e = cudaMalloc(p, bytes ? bytes : 1);
        if (e == cudaErrorMemoryAllocation) {
            cudaGetLastError();
            cudaMemPoolTrimTo(mp, 0);
            e = cudaMalloc(p, bytes ? bytes : 1);
        }
        if (e == cudaSuccess) {
            std::lock_guard<std::mutex> lock(mutex());
            direct().insert(*p);
        }
        return e;
    }
    cudaError_t e = cudaMallocFromPoolAsync(p, bytes ? bytes : 1, mp, stream());
    if (e == cudaErrorMemoryAllocation) {
        // what the pool keeps unused may be what is missing
        cudaGetLastError();
        cudaDeviceSynchronize();
        cudaMemPoolTrimTo(mp, 0);
        e = cudaMallocFromPoolAsync(p, bytes ? bytes : 1, mp, stream());
    }
    return e;
}

void dev_free(void* p)
{
    if (!p) return;
    cudaPointerAttributes at{};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaPointerGetAttributes(&at, p) != cudaSuccess) {
        cudaGetLastError();
        return;
    }
    if (at.device != dev) cudaSetDevice(at.device);
    bool own = true;
    {
        std::lock_guard<std::mutex> lock(mutex());
        own = direct().erase(p) == 0;
    }
    if (own && pool()) {
        cudaDeviceSynchronize();
        cudaFreeAsync(p, nullptr);
    } else {
        cudaFree(p);
    }
    if (at.device != dev) cudaSetDevice(dev);
}

cudaError_t pinned_malloc(void** p, size_t bytes)
{
    *p = nullptr;
    if (bytes > kPinnedBlock) return cudaErrorInvalidValue;
    {
        std::lock_guard<std::mutex> lock(mutex());
        if (!pinned().empty()) {
            *p = pinned().back();
            pinned().pop_back();
            return cudaSuccess;
        }
    }
    return cudaHostAlloc(p, kPinnedBlock, cudaHostAllocPortable);
}

void pinned_free(void* p)
{
    if (!p) return;
    {
        std::lock_guard<std::mutex> lock(mutex());
        if (pinned().size() < kPinned) {
            pinned().push_back(p);
            return;
        }
    }
    cudaFreeHost(p);
}

}  // namespace rg
