// scratch.cuh -- device memory that the library keeps between calls: one buffer per (device, stream) and kind of call, so that
// calls on different streams never share one.
//
//   which stream   told apart by its number (cudaStreamGetId), which no later stream is given again.  A handle would not do:
//                  cudaStreamPerThread is one handle for a stream in every thread, and a destroyed stream's handle can come back
//                  while its last work still runs.  Only a stream under capture, where its number may not be asked for, is known by
//                  its handle: the last stream that called with it.
//   the lock       a device's, held by the caller until the launches that use the buffer are enqueued: another thread on the same
//                  stream neither frees it in between nor puts its own launches there.
//   capture        nothing is allocated for a stream that is being captured, but the buffer that it has is used; a graph then
//                  holds its address, so it is neither freed nor given to another stream until release().
//   bound          16 streams per device; a 17th takes the buffer of one that has not called for a while (a program that uses
//                  17 in turn does not free and allocate on every call), or gets none: the caller has a kernel that needs none.
// cudaFree waits for the device, so nothing in flight reads what is freed.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <mutex>
#include <thread>
#include <vector>

namespace b200 {

// Zeroes new memory of the current device, complete on return, without a wait for any stream of the caller: on a stream of the library's own,
// one per device, made when first needed (making one per call took milliseconds).
inline bool zero_new_memory(void *p, size_t bytes) {
    static std::mutex mu;
    static cudaStream_t own[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev >= 64) return false;
    std::lock_guard<std::mutex> lock(mu);
    if (!own[dev] && cudaStreamCreateWithFlags(&own[dev], cudaStreamNonBlocking) != cudaSuccess) {
        own[dev] = nullptr;
        return false;
    }
    return cudaMemsetAsync(p, 0, bytes, own[dev]) == cudaSuccess && cudaStreamSynchronize(own[dev]) == cudaSuccess;
}

class StreamScratch {
public:
    // steps: a buffer that has become too small grows by half at least -- for calls whose need rises a little from one to the next.  (What is in
    // a buffer is whatever was there: the kernels write before they read.)
    explicit StreamScratch(bool steps) : steps_(steps) {}

    struct Lease {
        void *ptr = nullptr;                        // nullptr: none to be had
        std::unique_lock<std::mutex> lock;
    };

    // At least `bytes` of device memory, 256-byte aligned.
    Lease get(size_t bytes, cudaStream_t st, bool reserve = false) {
        Lease lease;
        int dev = 0;
        unsigned long long id = 0;
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        if (cudaGetDevice(&dev) != cudaSuccess || dev >= DEVICES || cudaStreamIsCapturing(st, &cap) != cudaSuccess ||
            (cap == cudaStreamCaptureStatusNone && cudaStreamGetId(st, &id) != cudaSuccess)) {
            (void)cudaGetLastError();
            return lease;
        }
        const bool capturing = cap != cudaStreamCaptureStatusNone;
        const std::thread::id thread = st == cudaStreamPerThread ? std::this_thread::get_id() : std::thread::id();
        Device &d = devices_[dev];
        lease.lock = std::unique_lock<std::mutex>(d.mu);
        Buffer *b = nullptr;
        for (size_t i = 0; i < d.n; ++i) {
            Buffer &x = d.buffers[i];
            const bool called = x.known && x.handle == st && x.thread == thread;
            if (capturing ? called : x.stream == id) b = &x;
            else if (called) x.known = false;        // a stream that is gone
        }
        if (!b || b->bytes < bytes) {
            if (capturing) return lease;
            if (!b) {
                if (d.n < STREAMS) {
                    b = &d.buffers[d.n++];
                } else {
                    for (auto &x : d.buffers)
                        if (!x.reserved && !x.in_graph && x.used + IDLE_CALLS <= d.calls && (!b || x.used < b->used)) b = &x;
                    if (!b) return lease;
                }
            }
            allocate(d, *b, id, bytes);
        }
        b->known = true;
        b->handle = st;
        b->thread = thread;
        b->used = ++d.calls;
        b->in_graph |= capturing;
        b->reserved |= reserve;
        lease.ptr = b->ptr;
        return lease;
    }

    // Frees everything, on every device.  Leaves the current device as it is.
    void release() {
        int now = 0;
        const bool have = cudaGetDevice(&now) == cudaSuccess;
        for (int dev = 0; dev < DEVICES; ++dev) {
            Device &d = devices_[dev];
            std::lock_guard<std::mutex> lock(d.mu);
            if (d.n == 0) continue;
            if (have) (void)cudaSetDevice(dev);
            for (size_t i = 0; i < d.n; ++i) (void)cudaFree(d.buffers[i].ptr), d.buffers[i] = Buffer();
            for (void *p : d.retired) (void)cudaFree(p);
            d.n = 0;
            d.retired.clear();
        }
        if (have) (void)cudaSetDevice(now);
    }

private:
    static constexpr int DEVICES = 64;
    static constexpr size_t STREAMS = 16;
    static constexpr unsigned long long IDLE_CALLS = 64;        // of the device's other streams
    struct Buffer {
        unsigned long long stream = 0, used = 0;
        cudaStream_t handle = nullptr;              // with which the stream called last, and from which thread if that matters
        std::thread::id thread;
        void *ptr = nullptr;
        size_t bytes = 0;
        bool known = false, reserved = false, in_graph = false;
    };
    struct Device {
        std::mutex mu;
        Buffer buffers[STREAMS];
        size_t n = 0;
        std::vector<void *> retired;                // outgrown, but a graph holds the address
        unsigned long long calls = 0;
    };

    void allocate(Device &d, Buffer &b, unsigned long long id, size_t bytes) {
        // another stream may be under capture: allocating is no part of that
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        (void)cudaThreadExchangeStreamCaptureMode(&mode);
        if (b.in_graph) retire(d, b.ptr);
        else (void)cudaFree(b.ptr);
        const bool same = b.stream == id, reserved = same && b.reserved;
        const size_t exact = bytes;
        if (steps_ && same && bytes < b.bytes + b.bytes / 2) bytes = b.bytes + b.bytes / 2;
        b = Buffer();
        b.stream = id;
        b.reserved = reserved;
        if (cudaMalloc(&b.ptr, bytes) != cudaSuccess && (bytes == exact || cudaMalloc(&b.ptr, bytes = exact) != cudaSuccess)) b.ptr = nullptr;
        if (b.ptr) b.bytes = bytes;
        else (void)cudaGetLastError();
        (void)cudaThreadExchangeStreamCaptureMode(&mode);
    }

    static void retire(Device &d, void *p) {
        try {
            d.retired.push_back(p);
        } catch (...) {                             // no memory on the host for the note: the buffer stays until the process ends
        }
    }

    const bool steps_;
    Device devices_[DEVICES];
};

}  // namespace b200
