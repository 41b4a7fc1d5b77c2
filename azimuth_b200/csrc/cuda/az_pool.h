// Device scratch and private streams that outlive a call.
//
// cudaMalloc and cudaFree wait for the device and take from tens of
// microseconds to several milliseconds each (a build allocates about a hundred
// buffers); a stream-ordered pool hands the same memory to the next call.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

namespace az {

// Memory of the current device's pool, usable by work on `st` from here on
// (and by other streams once they are ordered after `st`).  The pool keeps at
// most kPoolKept unused bytes across synchronisations; the rest goes back to
// the driver.  Safe with several threads and streams.
constexpr size_t kPoolKept = (size_t)2 << 30;
// Larger buffers are cudaMalloc's: the pool maps new memory at 7.3 ms per GiB
// and cannot keep much of a wave of tens of millions of samples, while
// cudaMalloc and cudaFree take 0.4 ms each for 128 MiB (the pool's growth 0.95)
// and 0.9 ms for 1 GiB.  A scene's queues live as long as the scene; what comes
// and goes with a call is smaller (one-shot image of 230 k samples: 48 MB the
// largest, a build of 1.3 M triangles: 62 MB).
constexpr size_t kPoolLargest = (size_t)128 << 20;
cudaError_t PoolAlloc(void **p, size_t bytes, cudaStream_t st);
// cudaMalloc, tried again after the pool has given back what it keeps unused.
cudaError_t DeviceAlloc(void **p, size_t bytes);
// Bytes that the current device's pool keeps unused (cudaMemGetInfo counts them as taken).
size_t PoolUnused();
// Waits for the current device and gives back all that is kept on it: the pool's unused memory and the idle streams.
cudaError_t PoolRelease();
// Gives memory back once the work queued on `st` so far has finished; no
// stream: when nothing uses the memory any more.
void PoolFree(void *p, cudaStream_t st);

// An array of the pool that lives as long as this object, used on one stream.
template <typename T>
struct PoolBuf {
    T *p = nullptr;
    cudaStream_t st = nullptr;
    PoolBuf() = default;
    PoolBuf(const PoolBuf &) = delete;
    PoolBuf &operator=(const PoolBuf &) = delete;
    ~PoolBuf() {
        if (p) PoolFree(p, st);
    }
    cudaError_t alloc(size_t n, cudaStream_t s) {
        st = s;
        return PoolAlloc((void **)&p, (n ? n : 1) * sizeof(T) + 16, s);
    }
};

// A blocking stream of the current device for one call (ordered after earlier
// work on the legacy default stream); at most kStreamsKept idle ones are kept
// per device.  ReleaseStream waits for the stream's work.
constexpr size_t kStreamsKept = 8;
cudaError_t AcquireStream(cudaStream_t *st);
void ReleaseStream(cudaStream_t st);

// A non-blocking stream with the two events that order it against a render's
// stream (it only ever runs after waiting on `fork`); idle ones are kept as above.
// ReleaseSide: when nothing runs on it any more.
struct SideStream {
    cudaStream_t stream = nullptr;
    cudaEvent_t fork = nullptr, join = nullptr;
};
cudaError_t AcquireSide(SideStream *s);
void ReleaseSide(const SideStream &s);

}  // namespace az
