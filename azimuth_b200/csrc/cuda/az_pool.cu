#include "az_pool.h"

#include <mutex>
#include <unordered_set>
#include <vector>

namespace az {
namespace {

constexpr int kMaxDevices = 64;

struct DevicePools {
    std::mutex mu;
    cudaMemPool_t pool[kMaxDevices] = {};
    std::vector<cudaStream_t> streams[kMaxDevices];
    std::vector<SideStream> sides[kMaxDevices];
    cudaStream_t idle[kMaxDevices] = {};   // takes the frees of memory that no work uses any more
    std::unordered_set<void *> direct;     // buffers of cudaMalloc
};

// Never destroyed: the driver may be gone when static destructors run.
DevicePools &Pools() {
    static DevicePools *p = new DevicePools();
    return *p;
}

cudaError_t PoolOf(int dev, cudaMemPool_t *out) {
    if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
    DevicePools &P = Pools();
    std::lock_guard<std::mutex> lock(P.mu);
    if (!P.pool[dev]) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t pool = nullptr;
        cudaError_t e = cudaMemPoolCreate(&pool, &props);
        if (e != cudaSuccess) return e;
        unsigned long long kept = kPoolKept;
        e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &kept);
        if (e != cudaSuccess) {
            cudaMemPoolDestroy(pool);
            return e;
        }
        P.pool[dev] = pool;
    }
    *out = P.pool[dev];
    return cudaSuccess;
}

}  // namespace

// What the pool keeps may be in the way of an allocation: gives it back once the
// frees queued on `st` and without a stream have finished.
static void Trim(int dev, cudaStream_t st) {
    cudaGetLastError();
    cudaStream_t idle = nullptr;
    cudaMemPool_t pool = nullptr;
    {
        DevicePools &P = Pools();
        std::lock_guard<std::mutex> lock(P.mu);
        if (dev < 0 || dev >= kMaxDevices || !P.pool[dev]) return;
        pool = P.pool[dev];
        idle = P.idle[dev];
    }
    if (idle) cudaStreamSynchronize(idle);
    if (st) cudaStreamSynchronize(st);
    cudaMemPoolTrimTo(pool, 0);
    cudaGetLastError();
}

static cudaError_t AllocTrimmed(void **p, size_t bytes, int dev, cudaStream_t st) {
    cudaError_t e = cudaMalloc(p, bytes);
    if (e == cudaErrorMemoryAllocation) {
        Trim(dev, st);
        e = cudaMalloc(p, bytes);
    }
    if (e != cudaSuccess) {
        *p = nullptr;
        cudaGetLastError();
    }
    return e;
}

cudaError_t DeviceAlloc(void **p, size_t bytes) {
    *p = nullptr;
    int dev = 0;
    const cudaError_t e = cudaGetDevice(&dev);
    return e == cudaSuccess ? AllocTrimmed(p, bytes, dev, nullptr) : e;
}

cudaError_t PoolAlloc(void **p, size_t bytes, cudaStream_t st) {
    *p = nullptr;
    int dev = 0;
    cudaMemPool_t pool = nullptr;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess && bytes > kPoolLargest) {
        e = AllocTrimmed(p, bytes, dev, st);
        if (e == cudaSuccess) {
            DevicePools &P = Pools();
            std::lock_guard<std::mutex> lock(P.mu);
            P.direct.insert(*p);
        }
        return e;
    }
    if (e == cudaSuccess) e = PoolOf(dev, &pool);
    if (e != cudaSuccess) return e;
    e = cudaMallocFromPoolAsync(p, bytes, pool, st);
    if (e == cudaErrorMemoryAllocation) {
        Trim(dev, st);
        e = cudaMallocFromPoolAsync(p, bytes, pool, st);
    }
    if (e != cudaSuccess) {
        *p = nullptr;
        cudaGetLastError();
    }
    return e;
}

size_t PoolUnused() {
    int dev = 0;
    cudaMemPool_t pool = nullptr;
    if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < kMaxDevices) {
        DevicePools &P = Pools();
        std::lock_guard<std::mutex> lock(P.mu);
        pool = P.pool[dev];
    }
    unsigned long long reserved = 0, used = 0;
    if (!pool || cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &reserved) != cudaSuccess ||
        cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return reserved > used ? (size_t)(reserved - used) : 0;
}

cudaError_t PoolRelease() {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e != cudaSuccess || dev < 0 || dev >= kMaxDevices) return e;
    std::vector<cudaStream_t> streams;
    std::vector<SideStream> sides;
    {
        DevicePools &P = Pools();
        std::lock_guard<std::mutex> lock(P.mu);
        streams.swap(P.streams[dev]);
        sides.swap(P.sides[dev]);
    }
    for (cudaStream_t s : streams) cudaStreamDestroy(s);
    for (const SideStream &s : sides) {
        cudaEventDestroy(s.fork);
        cudaEventDestroy(s.join);
        cudaStreamDestroy(s.stream);
    }
    Trim(dev, nullptr);
    return cudaSuccess;
}

void PoolFree(void *p, cudaStream_t st) {
    if (!p) return;
    DevicePools &P = Pools();
    {
        std::lock_guard<std::mutex> lock(P.mu);
        if (P.direct.erase(p) == 0) {
            // Not on the legacy default stream: a free queued there would break a
            // capture that another thread has open on a stream of its own.
            int dev = 0;
            if (!st && cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < kMaxDevices) {
                if (!P.idle[dev] && cudaStreamCreateWithFlags(&P.idle[dev], cudaStreamNonBlocking) != cudaSuccess) {
                    P.idle[dev] = nullptr;
                    cudaGetLastError();
                }
                st = P.idle[dev];
            }
            cudaFreeAsync(p, st);
            return;
        }
    }
    cudaFree(p);   // waits for the device, as the work on `st` needs
}

cudaError_t AcquireStream(cudaStream_t *st) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < kMaxDevices) {
        DevicePools &P = Pools();
        std::lock_guard<std::mutex> lock(P.mu);
        if (!P.streams[dev].empty()) {
            *st = P.streams[dev].back();
            P.streams[dev].pop_back();
            return cudaSuccess;
        }
    }
    return cudaStreamCreate(st);
}

void ReleaseStream(cudaStream_t st) {
    cudaStreamSynchronize(st);
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < kMaxDevices) {
        DevicePools &P = Pools();
        std::lock_guard<std::mutex> lock(P.mu);
        if (P.streams[dev].size() < kStreamsKept) {
            P.streams[dev].push_back(st);
            return;
        }
    }
    cudaStreamDestroy(st);
}

cudaError_t AcquireSide(SideStream *s) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < kMaxDevices) {
        DevicePools &P = Pools();
        std::lock_guard<std::mutex> lock(P.mu);
        if (!P.sides[dev].empty()) {
            *s = P.sides[dev].back();
            P.sides[dev].pop_back();
            return cudaSuccess;
        }
    }
    SideStream n;
    e = cudaStreamCreateWithFlags(&n.stream, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&n.fork, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&n.join, cudaEventDisableTiming);
    if (e != cudaSuccess) {
        if (n.fork) cudaEventDestroy(n.fork);
        if (n.stream) cudaStreamDestroy(n.stream);
        return e;
    }
    *s = n;
    return cudaSuccess;
}

void ReleaseSide(const SideStream &s) {
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < kMaxDevices) {
        DevicePools &P = Pools();
        std::lock_guard<std::mutex> lock(P.mu);
        if (P.sides[dev].size() < kStreamsKept) {
            P.sides[dev].push_back(s);
            return;
        }
    }
    cudaEventDestroy(s.fork);
    cudaEventDestroy(s.join);
    cudaStreamDestroy(s.stream);
}

}  // namespace az
