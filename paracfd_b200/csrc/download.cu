// download.cu -- large device-to-host copies into ordinary (pageable) memory.
//
// A plain copy into pageable memory goes through the driver's staging buffer on one host thread,
// which also takes the page faults of a freshly allocated destination: 54 ms for the 310 MB of
// velocity and pressure on the 16 M-cell grid (6 GB/s), 18 ms with this.  Here up to eight host threads take 1 MiB
// pieces in turn: each stages its piece in pinned memory of its own (two pieces in flight) and
// copies it on, so the faults and copies run side by side.  Each thread has a stream of its own that
// waits for what the caller's stream holds: the caller's may be cudaStreamPerThread, which in
// another thread names another stream.  Pinned pieces and streams belong to the system and go with
// it.  Copies below kThreadedCopy, where starting threads costs more than it gives, copies into
// pinned memory and copies of a stream that is being captured stay plain.
#include "pcfd_internal.h"

#include <algorithm>
#include <atomic>
#include <cstring>
#include <thread>

namespace pcfd
{
    namespace
    {
        constexpr size_t kThreadedCopy = size_t(8) << 20, kPiece = size_t(1) << 20;
        constexpr int kMostThreads = 8;
    }

    struct Download
    {
        int threads = 0;
        char* pinned = nullptr;                         // [threads][2][kPiece]
        cudaStream_t stream[kMostThreads] = {};
        cudaEvent_t ready[kMostThreads][2] = {};
        cudaEvent_t produced = nullptr;                 // what the caller's stream held before the copies
        ~Download()
        {
            for (cudaStream_t one : stream)
                if (one) cudaStreamDestroy(one);
            for (auto& pair : ready)
                for (cudaEvent_t e : pair)
                    if (e) cudaEventDestroy(e);
            if (produced) cudaEventDestroy(produced);
            if (pinned) cudaFreeHost(pinned);
        }
    };

    namespace
    {
        // the system's device while this lives, then the thread's own again
        struct OnDevice
        {
            int before = 0;
            bool changed = false;
            explicit OnDevice(int device)
            {
                cuda_check(cudaGetDevice(&before), "current device");
                changed = before != device;
                if (changed) cuda_check(cudaSetDevice(device), "set device");
            }
            ~OnDevice()
            {
                if (changed) cudaSetDevice(before);
            }
        };

        // the system's staging, made on its first large copy; false when the host has none to give
        bool staging(System& s)
        {
            if (s.download) return s.download->threads > 1;
            auto d = std::make_shared<Download>();
            d->threads = int(std::min<unsigned>(kMostThreads, std::max(1u, std::thread::hardware_concurrency())));
            bool made = d->threads > 1 && cudaMallocHost(&d->pinned, size_t(d->threads) * 2 * kPiece) == cudaSuccess &&
                        cudaEventCreateWithFlags(&d->produced, cudaEventDisableTiming) == cudaSuccess;
            for (int t = 0; t < d->threads && made; ++t)
            {
                made = cudaStreamCreateWithFlags(&d->stream[t], cudaStreamNonBlocking) == cudaSuccess;
                for (cudaEvent_t& e : d->ready[t]) made = made && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
            }
            if (!made)
            {
                cudaGetLastError();
                d = std::make_shared<Download>();
                d->threads = 1;
            }
            s.download = std::move(d);
            return s.download->threads > 1;
        }
    }

    bool threaded_download(System& s, void* dst, const void* src, size_t bytes)
    {
        if (bytes < kThreadedCopy) return false;
        cudaPointerAttributes where{};
        if (cudaPointerGetAttributes(&where, dst) != cudaSuccess) cudaGetLastError();
        else if (where.type != cudaMemoryTypeUnregistered) return false;
        cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(s.stream, &capture) != cudaSuccess) cudaGetLastError();
        if (capture != cudaStreamCaptureStatusNone) return false;
        // streams and events are made and recorded on the system's device, whichever this thread uses
        const OnDevice on(s.device);
        if (!staging(s)) return false;
        Download& d = *s.download;
        const size_t pieces = (bytes + kPiece - 1) / kPiece;
        const int want = int(std::min<size_t>(size_t(d.threads), pieces));
        // recorded by the calling thread, which is the one that enqueued the work
        cuda_check(cudaEventRecord(d.produced, s.stream), "download event");
        for (int t = 0; t < want; ++t) cuda_check(cudaStreamWaitEvent(d.stream[t], d.produced, 0), "download wait");
        std::atomic<size_t> next{0};
        std::atomic<int> failed{int(cudaSuccess)};
        auto work = [&](int t) {
            auto check = [&](cudaError_t e) {
                if (e != cudaSuccess) failed.store(int(e));
                return e == cudaSuccess;
            };
            if (t > 0 && !check(cudaSetDevice(s.device))) return;
            char* const stage = d.pinned + size_t(t) * 2 * kPiece;
            size_t held[2] = {pieces, pieces};           // piece in flight per buffer
            auto size = [&](size_t p) { return std::min(kPiece, bytes - p * kPiece); };
            auto start = [&](int b) {
                held[b] = failed.load() ? pieces : next.fetch_add(1);
                if (held[b] >= pieces) { held[b] = pieces; return; }
                if (!check(cudaMemcpyAsync(stage + size_t(b) * kPiece, static_cast<const char*>(src) + held[b] * kPiece, size(held[b]),
                                           cudaMemcpyDeviceToHost, d.stream[t])) ||
                    !check(cudaEventRecord(d.ready[t][b], d.stream[t])))
                    held[b] = pieces;
            };
            start(0);
            for (int b = 0; held[b] < pieces; b ^= 1)
            {
                start(b ^ 1);
                if (!check(cudaEventSynchronize(d.ready[t][b]))) return;
                std::memcpy(static_cast<char*>(dst) + held[b] * kPiece, stage + size_t(b) * kPiece, size(held[b]));
            }
        };
        std::vector<std::thread> helpers;
        try
        {
            helpers.reserve(size_t(want));
            for (int t = 1; t < want; ++t) helpers.emplace_back(work, t);
        }
        catch (...)
        {
            // no memory or no thread for more: those there are take all pieces
        }
        work(0);
        for (std::thread& h : helpers) h.join();
        // nothing may still write the pinned pieces or read the source after an error
        if (failed.load())
            for (int t = 0; t < want; ++t) cudaStreamSynchronize(d.stream[t]);
        cuda_check(cudaError_t(failed.load()), "device to host");
        return true;
    }
}
