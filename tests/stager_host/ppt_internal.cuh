// A stand-in for the CUDA runtime, for csrc/staging.cu on a machine without a
// GPU: "device" memory is host memory, a stream is a thread that runs its
// operations in order, an event is complete once its last record has run.
#pragma once
#include <atomic>
#include <condition_variable>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <memory>
#include <mutex>
#include <string>
#include <thread>

#include "ppt.h"

using cudaError_t = int;
constexpr cudaError_t cudaSuccess = 0, cudaErrorMemoryAllocation = 2, cudaErrorUnknown = 999;
enum { cudaMemcpyHostToDevice, cudaMemcpyDeviceToHost };
constexpr int cudaEventDisableTiming = 0, cudaHostAllocDefault = 0;

struct FakeMark {                 // one record of an event
    std::mutex m;
    std::condition_variable cv;
    bool done = false;
    cudaError_t error = 0;
    void complete(cudaError_t e) {
        std::lock_guard<std::mutex> lock(m);
        done = true;
        error = e;
        cv.notify_all();
    }
    cudaError_t wait() {
        std::unique_lock<std::mutex> lock(m);
        cv.wait(lock, [&] { return done; });
        return error;
    }
};
struct FakeEvent {
    std::mutex m;
    std::shared_ptr<FakeMark> mark;
    std::shared_ptr<FakeMark> last() {
        std::lock_guard<std::mutex> lock(m);
        return mark;
    }
};
struct FakeStream {
    std::mutex m;
    std::condition_variable cv;
    std::deque<std::function<void()>> ops;
    bool stop = false;
    std::thread worker{[this] {
        for (;;) {
            std::function<void()> op;
            {
                std::unique_lock<std::mutex> lock(m);
                cv.wait(lock, [&] { return stop || !ops.empty(); });
                if (ops.empty()) return;
                op = std::move(ops.front());
                ops.pop_front();
            }
            op();
        }
    }};
    void add(std::function<void()> op) {
        std::lock_guard<std::mutex> lock(m);
        ops.push_back(std::move(op));
        cv.notify_all();
    }
    ~FakeStream() {
        {
            std::lock_guard<std::mutex> lock(m);
            stop = true;
            cv.notify_all();
        }
        worker.join();
    }
};
using cudaStream_t = FakeStream*;
using cudaEvent_t = FakeEvent*;

inline std::atomic<int> fake_copies_left{1 << 30};   // memcpys until one is refused
inline std::atomic<int> fake_in_flight{0};           // queued memcpys that have not run
inline std::atomic<const void*> fake_bad_source{nullptr};   // a copy that reads it fails when it runs

inline cudaError_t cudaGetDevice(int* d) { *d = 0; return 0; }
inline cudaError_t cudaSetDevice(int) { return 0; }
inline cudaError_t cudaHostAlloc(char** p, size_t n, int) { *p = static_cast<char*>(std::malloc(n)); return *p ? 0 : 2; }
inline cudaError_t cudaFreeHost(void* p) { std::free(p); return 0; }
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, int) { *e = new FakeEvent; return 0; }
inline cudaError_t cudaEventDestroy(cudaEvent_t e) { delete e; return 0; }
inline thread_local cudaError_t fake_stream_error = 0;       // of the stream's thread: its last copy's
inline cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    auto mark = std::make_shared<FakeMark>();
    {
        std::lock_guard<std::mutex> lock(e->m);
        e->mark = mark;
    }
    s->add([mark] { mark->complete(fake_stream_error); });
    return 0;
}
inline cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    auto mark = e->last();
    return mark ? mark->wait() : 0;
}
inline cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, int) {
    auto mark = e->last();
    if (mark) s->add([mark] { mark->wait(); });
    return 0;
}
inline cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    FakeEvent e;
    cudaEventRecord(&e, s);
    cudaEventSynchronize(&e);
    return 0;
}
inline cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, int, cudaStream_t s) {
    if (fake_copies_left.fetch_sub(1) <= 0) return cudaErrorUnknown;
    fake_in_flight.fetch_add(1);
    s->add([=] {
        fake_stream_error = src == fake_bad_source.load() ? cudaErrorUnknown : 0;
        if (!fake_stream_error) std::memcpy(dst, src, n);
        fake_in_flight.fetch_sub(1);
    });
    return 0;
}

namespace ppt {
inline int fail(int code, const std::string&) { return code; }
inline int cuda_fail(cudaError_t, const char*) { return PPT_ERR_CUDA; }
}  // namespace ppt
#define PPT_CUDA_TRY(expr)                                  \
    do {                                                    \
        const cudaError_t _e = (expr);                      \
        if (_e != cudaSuccess) return PPT_ERR_CUDA;         \
    } while (0)
