// Large downloads and device buffers against a stand-in for the CUDA runtime: no GPU, no driver.
//
// The stand-in keeps what the checks are about.  Devices are numbers; a thread has a current device.  A
// stream is a queue of actions that run only when something waits for them; cudaStreamPerThread
// names the calling thread's own queue and the null stream the current device's.  An event belongs
// to the device it was made on and may be recorded on that device's streams only.
#include "../../paracfd_b200/csrc/download.cu"

#include <cstdio>
#include <cstdlib>
#include <deque>
#include <functional>
#include <map>
#include <mutex>
#include <new>

namespace
{
    struct Queue
    {
        int device = 0;
        std::deque<std::function<void()>> pending;
        void drain()
        {
            while (!pending.empty())
            {
                auto action = std::move(pending.front());
                pending.pop_front();
                action();
            }
        }
    };
    struct Event
    {
        int device = 0;
        Queue* queue = nullptr;      // recorded on; a wait runs all of its queue (later actions may run early)
    };
    thread_local int current = 0;
    std::map<std::pair<int, std::thread::id>, Queue> per_thread;
    std::map<int, Queue> legacy;
    bool fail_device_memory = false;
    thread_local int allocations_left = -1;      // of this thread's operator new; < 0: no limit
    // one call of the stand-in at a time; its own allocations do not count
    struct Call
    {
        static std::recursive_mutex& lock() { static std::recursive_mutex one; return one; }
        std::lock_guard<std::recursive_mutex> guard{lock()};
        int left = allocations_left;
        Call() { allocations_left = -1; }
        ~Call() { allocations_left = left; }
    };

    Queue& queue_of(cudaStream_t stream)
    {
        Queue* q;
        if (stream == cudaStreamPerThread) q = &per_thread[{current, std::this_thread::get_id()}];
        else if (!stream || stream == cudaStreamLegacy) q = &legacy[current];
        else return *reinterpret_cast<Queue*>(stream);
        q->device = current;
        return *q;
    }
}

extern "C"
{
    cudaError_t cudaSetDevice(int device) { current = device; return cudaSuccess; }
    cudaError_t cudaGetDevice(int* device) { *device = current; return cudaSuccess; }
    cudaError_t cudaGetLastError() { return cudaSuccess; }
    const char* cudaGetErrorString(cudaError_t) { return "stand-in error"; }
    cudaError_t cudaMalloc(void** p, size_t bytes)
    {
        if (fail_device_memory) return cudaErrorMemoryAllocation;
        *p = std::malloc(bytes);
        return cudaSuccess;
    }
    cudaError_t cudaFree(void* p) { std::free(p); return cudaSuccess; }
    // on the null stream, and done when something waits for it: a copy out of ordinary memory returns once
    // the source has been staged, a memset at once
    cudaError_t cudaMemset(void* p, int value, size_t bytes)
    {
        const Call call;
        legacy[current].pending.push_back([=] { std::memset(p, value, bytes); });
        return cudaSuccess;
    }
    cudaError_t cudaMemcpy(void* to, const void* from, size_t bytes, cudaMemcpyKind)
    {
        const Call call;
        const std::vector<char> staged(static_cast<const char*>(from), static_cast<const char*>(from) + bytes);
        legacy[current].pending.push_back([=] { std::memcpy(to, staged.data(), bytes); });
        return cudaSuccess;
    }
    cudaError_t cudaHostAlloc(void** p, size_t bytes, unsigned) { *p = std::malloc(bytes); return cudaSuccess; }
    cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
    cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) { a->type = cudaMemoryTypeUnregistered; return cudaSuccess; }
    cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned)
    {
        const Call call;
        auto* q = new Queue;
        q->device = current;
        *s = reinterpret_cast<cudaStream_t>(q);
        return cudaSuccess;
    }
    cudaError_t cudaStreamDestroy(cudaStream_t s) { delete reinterpret_cast<Queue*>(s); return cudaSuccess; }
    cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) { *s = cudaStreamCaptureStatusNone; return cudaSuccess; }
    cudaError_t cudaStreamSynchronize(cudaStream_t s)
    {
        const Call call;
        queue_of(s).drain();
        return cudaSuccess;
    }
    cudaError_t cudaMemcpyAsync(void* to, const void* from, size_t bytes, cudaMemcpyKind, cudaStream_t s)
    {
        const Call call;
        queue_of(s).pending.push_back([=] { std::memcpy(to, from, bytes); });
        return cudaSuccess;
    }
    cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned)
    {
        const Call call;
        auto* event = new Event;
        event->device = current;
        *e = reinterpret_cast<cudaEvent_t>(event);
        return cudaSuccess;
    }
    cudaError_t cudaEventDestroy(cudaEvent_t e) { delete reinterpret_cast<Event*>(e); return cudaSuccess; }
    cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s)
    {
        const Call call;
        Queue& q = queue_of(s);
        Event& event = *reinterpret_cast<Event*>(e);
        if (event.device != q.device) return cudaErrorInvalidResourceHandle;
        event.queue = &q;
        return cudaSuccess;
    }
    cudaError_t cudaEventSynchronize(cudaEvent_t e)
    {
        const Call call;
        Event& event = *reinterpret_cast<Event*>(e);
        if (event.queue) event.queue->drain();
        return cudaSuccess;
    }
    cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned)
    {
        const Call call;
        Queue* from = reinterpret_cast<Event*>(e)->queue;
        if (from) queue_of(s).pending.push_back([from] { from->drain(); });
        return cudaSuccess;
    }
}

namespace pcfd
{
    System::~System() {}
}

namespace
{
    constexpr size_t kBytes = (size_t(22) << 20) + 12345;      // 23 pieces, a ragged last one

    // A download of a system on `device` and `stream` by a thread whose current device is `from`, right
    // after a kernel that writes the data was enqueued.  limit >= 0: host allocations that
    // thread has left; then an error is an answer too, but not another current device or other data.
    bool download(pcfd::System& s, int device, cudaStream_t stream, int from, int seed, int limit = -1)
    {
        std::vector<unsigned char> source(kBytes, 0), result(kBytes, 0xEE);
        current = device;
        queue_of(stream).pending.push_back([&] { for (size_t i = 0; i < kBytes; ++i) source[i] = static_cast<unsigned char>(i * 7 + seed); });
        current = from;
        s.device = device;
        s.stream = stream;
        bool done = false;
        allocations_left = limit;
        try
        {
            done = pcfd::threaded_download(s, result.data(), source.data(), kBytes);
            allocations_left = -1;
        }
        catch (const std::bad_alloc&)
        {
            allocations_left = -1;
            if (limit < 0) throw;
        }
        if (current != from) { std::printf("current device %d, was %d\n", current, from); return false; }
        if (!done) { queue_of(stream).drain(); std::puts("not threaded"); return limit >= 0; }
        if (source[5] != static_cast<unsigned char>(35 + seed) || result != source) { std::puts("stale data"); return false; }
        return true;
    }
}

void* operator new(size_t bytes)
{
    if (allocations_left == 0) throw std::bad_alloc();
    if (allocations_left > 0) --allocations_left;
    if (void* p = std::malloc(bytes)) return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

int main(int argc, char** argv)
{
    const std::string check = argc > 1 ? argv[1] : "";
    try
    {
        pcfd::System s;
        if (check == "per-thread stream") return download(s, 0, cudaStreamPerThread, 0, 1) && download(s, 0, cudaStreamPerThread, 0, 2) ? 0 : 1;
        if (check == "other device")
        {
            Queue own;
            own.device = 1;
            const cudaStream_t stream = reinterpret_cast<cudaStream_t>(&own);
            return download(s, 1, stream, 0, 1) && download(s, 1, stream, 1, 2) && download(s, 1, stream, 0, 3) ? 0 : 1;
        }
        if (check == "failed thread start")
        {
            Queue own;
            const cudaStream_t stream = reinterpret_cast<cudaStream_t>(&own);
            bool ok = download(s, 0, stream, 0, 1);
            for (int limit = 0; limit < 12 && ok; ++limit) ok = download(s, 0, stream, 0, 2 + limit, limit);
            return ok ? 0 : 1;
        }
        if (check == "uploads complete")
        {
            // what a stream that does not wait for the null stream would read right after the call
            pcfd::DBuf<int> buffer;
            buffer.upload(std::vector<int>(1000, 7));
            if (buffer.p[0] != 7 || buffer.p[999] != 7) { std::puts("upload not complete"); return 1; }
            buffer.alloc(1000);
            if (buffer.p[0] != 0 || buffer.p[999] != 0) { std::puts("clearing not complete"); return 1; }
            return 0;
        }
        if (check == "failed allocation")
        {
            pcfd::DBuf<float> buffer;
            fail_device_memory = true;
            try { buffer.alloc(100); std::puts("no error"); return 1; }
            catch (const pcfd::Error& e) { if (e.status != PCFD_OUT_OF_MEMORY) return 1; }
            if (buffer.n != 0 || buffer.p) { std::printf("%zu entries after a failed allocation\n", buffer.n); return 1; }
            fail_device_memory = false;
            buffer.alloc(100);
            return buffer.n == 100 && buffer.p ? 0 : 1;
        }
    }
    catch (const std::exception& e) { std::printf("error: %s\n", e.what()); return 1; }
    std::puts("unknown check");
    return 2;
}
