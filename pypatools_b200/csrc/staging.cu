// Host <-> device copies through a ring of pinned buffers, with the host side
// of every piece moved by a pool of threads.
//
// The arrays a track starts from and the histories it returns are ordinary
// (pageable) host memory: a device copy from or into it runs at 10 GB/s, and
// pinning it costs more than the copy.  An upload's pieces are claimed by the
// caller and whichever threads are awake, each copying its piece into a pinned
// slot and queueing that slot's copy; a download's pieces land in slots and are
// copied out by the pool.  What bounds it, on the 16-core host of a B200: PCIe
// (55 GB/s), the memory (about 50 GB/s of copying), one thread (17 GB/s), and
// waking a sleeping thread (up to 0.1 ms): so the caller starts without waiting
// for the others, and threads look for more work for a while before they sleep.
// The stores go past the cache: the GPU reads lines that are dirty in it at
// 17 GB/s, and landed histories are more than it holds.  Measured, a pool that
// copied through it and was woken piece by piece -> this: upload of 24 / 120 /
// 480 MB 2.8 / 5.6 / 17.1 -> 0.67 / 2.9 / 10.8 ms, download 2.7 / 5.2 / 16.3 ->
// 0.59 / 2.7 / 9.9 ms.  The reference has no counterpart (its arrays never leave
// the host).
#include <semaphore.h>

#include <atomic>
#include <condition_variable>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <new>
#include <thread>
#include <vector>
#if defined(__x86_64__)
#include <emmintrin.h>
#endif

#include "ppt_internal.cuh"

namespace ppt {

constexpr int64_t kMinPiece = 256 << 10;
constexpr int64_t kStreamBytes = 1 << 20;    // copies beyond this bypass the cache
constexpr int64_t kBytesPerThread = 4 << 20; // an upload wakes a thread for every so many bytes
constexpr int kSpins = 2000;                 // ~0.1 ms of looking for work before a thread sleeps

static inline void spin_pause() {
#if defined(__x86_64__)
    _mm_pause();
#endif
}

static void copy_bytes(char* dst, const char* src, int64_t bytes, bool stream) {
#if defined(__x86_64__)
    if (stream && bytes >= 4096) {
        const int64_t head = (16 - (int64_t)(reinterpret_cast<uintptr_t>(dst) & 15)) & 15;
        std::memcpy(dst, src, (size_t)head);
        int64_t i = head;
        for (; i + 64 <= bytes; i += 64) {
            const __m128i* from = reinterpret_cast<const __m128i*>(src + i);
            __m128i* to = reinterpret_cast<__m128i*>(dst + i);
            const __m128i a = _mm_loadu_si128(from), b = _mm_loadu_si128(from + 1);
            const __m128i c = _mm_loadu_si128(from + 2), d = _mm_loadu_si128(from + 3);
            _mm_stream_si128(to, a);
            _mm_stream_si128(to + 1, b);
            _mm_stream_si128(to + 2, c);
            _mm_stream_si128(to + 3, d);
        }
        std::memcpy(dst + i, src + i, (size_t)(bytes - i));
        _mm_sfence();
        return;
    }
#endif
    (void)stream;
    std::memcpy(dst, src, (size_t)bytes);
}

struct StagerSlot {
    char* buf = nullptr;
    cudaEvent_t ev = nullptr;   // the slot's last copy
    bool busy = false;          // a download's piece, until it has landed
    uint64_t seq = 0;           // its number
    bool in_flight = false;     // an upload's copy is queued
};

struct StagerLanding {
    int slot;
    char* host;
    int64_t bytes;
    bool stream;
    std::thread::id caller;
};

// A queue of landings that never allocates: a slot is in it at most once.
struct StagerQueue {
    std::vector<StagerLanding> at;
    size_t first = 0, count = 0;
    bool empty() const { return count == 0; }
    void push(const StagerLanding& t) { at[(first + count++) % at.size()] = t; }
    StagerLanding pop() {
        const StagerLanding t = at[first];
        first = (first + 1) % at.size();
        --count;
        return t;
    }
};

struct StagerSleeper {
    sem_t sem;
    std::atomic<bool> asleep{false};
    StagerSleeper() { sem_init(&sem, 0, 0); }
    ~StagerSleeper() { sem_destroy(&sem); }
    StagerSleeper(const StagerSleeper&) = delete;
};

// The pieces of an upload, claimed one by one.
struct StagerUpload {
    char* dev = nullptr;
    const char* host = nullptr;
    int64_t bytes = 0, piece = 0;
    int first = 0;                          // slots first, first + 1, ... (around the ring)
    std::atomic<int> n{0};                  // pieces (idle threads look at it while the next upload sets it)
    bool stream = false;
    std::atomic<int> next{0}, done{0};
    std::atomic<int> error{0};
};

}  // namespace ppt

struct ppt_stager {
    int device = 0;
    int64_t slot_bytes = 0;
    cudaStream_t stream = nullptr;
    char* pinned = nullptr;
    std::vector<ppt::StagerSlot> slots;
    std::vector<std::thread> threads;       // the pool, and last the thread that waits for downloads
    int pool = 0;
    std::mutex ring;                        // one upload or download is being cut into pieces at a time
    ppt::StagerUpload up;
    std::mutex m;                           // the fields below and the slots' busy and seq
    ppt::StagerQueue arriving;              // device -> slot, in the order of the copies
    ppt::StagerQueue land;                  // slot -> host
    std::condition_variable arrival, done;
    // The pool joins without the mutex: threads woken one after the other through
    // it would queue for it.  A thread counts itself into `joined` before it looks
    // at up_open, and the caller closes up_open before it waits for `joined`.
    std::atomic<bool> up_open{false};       // pieces of `up` may be claimed
    std::atomic<int> joined{0};             // threads of the pool at it
    std::atomic<int> landings{0};           // entries of `land`
    std::atomic<bool> stop{false};
    std::unique_ptr<ppt::StagerSleeper[]> sleepers;   // one per thread of the pool
    bool stop_waiter = false;
    size_t next = 0;
    uint64_t queued = 0;                    // download pieces so far
    cudaError_t lost_error = cudaSuccess;
    std::map<std::thread::id, cudaError_t> errors;   // of the downloads of each caller, until its finish
};

namespace ppt {

static void claim_pieces(ppt_stager* S) {
    StagerUpload& U = S->up;
    for (;;) {
        const int i = U.next.fetch_add(1);
        if (i >= U.n) return;
        StagerSlot& slot = S->slots[(size_t)(U.first + i) % S->slots.size()];
        const int64_t a = i * U.piece, b = a + U.piece < U.bytes ? a + U.piece : U.bytes;
        copy_bytes(slot.buf, U.host + a, b - a, U.stream);
        cudaError_t e = cudaMemcpyAsync(U.dev + a, slot.buf, (size_t)(b - a), cudaMemcpyHostToDevice, S->stream);
        if (e == cudaSuccess) e = cudaEventRecord(slot.ev, S->stream);
        slot.in_flight = e == cudaSuccess;
        int none = 0;
        if (e != cudaSuccess) U.error.compare_exchange_strong(none, (int)e);
        U.done.fetch_add(1);
    }
}

static void wake(ppt_stager* S, int count) {
    for (int k = 0; k < S->pool && count > 0; ++k)
        if (S->sleepers[k].asleep.exchange(false)) {
            sem_post(&S->sleepers[k].sem);
            --count;
        }
}

// The first error among a caller's downloads; with S->m held.  (Without the
// memory to note it, it is everyone's: see ppt_stager_finish.)
static void note_error(ppt_stager* S, std::thread::id caller, cudaError_t e) {
    try {
        S->errors.emplace(caller, e);
    } catch (const std::exception&) {
        S->lost_error = e;
    }
}

// Downloads' copies finish in order: one thread waits for them, so that no
// thread of the pool is held by the GPU.
static void stager_waiter(ppt_stager* S) {
    cudaSetDevice(S->device);
    for (;;) {
        StagerLanding t;
        {
            std::unique_lock<std::mutex> lock(S->m);
            S->arrival.wait(lock, [&] { return S->stop_waiter || !S->arriving.empty(); });
            if (S->arriving.empty()) return;
            t = S->arriving.pop();
        }
        const cudaError_t e = cudaEventSynchronize(S->slots[t.slot].ev);
        const bool small = t.bytes <= kMinPiece;       // not worth handing over
        if (e == cudaSuccess && small) copy_bytes(t.host, S->slots[t.slot].buf, t.bytes, t.stream);
        std::lock_guard<std::mutex> lock(S->m);
        if (e == cudaSuccess && !small) {
            S->land.push(t);
            S->landings.fetch_add(1);
            wake(S, 1);
        } else {
            if (e != cudaSuccess) note_error(S, t.caller, e);
            S->slots[t.slot].busy = false;
            S->done.notify_all();
        }
    }
}

static void stager_worker(ppt_stager* S, int me) {
    cudaSetDevice(S->device);
    StagerSleeper& mine = S->sleepers[me];
    auto work = [&] { return S->up_open.load() || S->landings.load() > 0 || S->stop.load(); };
    for (;;) {
        if (S->up_open.load()) {
            S->joined.fetch_add(1);
            if (S->up_open.load()) claim_pieces(S);
            S->joined.fetch_sub(1);
        }
        if (S->landings.load() > 0) {
            StagerLanding t;
            bool have = false;
            {
                std::lock_guard<std::mutex> lock(S->m);
                if (!S->land.empty()) {
                    t = S->land.pop();
                    S->landings.fetch_sub(1);
                    have = true;
                }
            }
            if (have) {
                copy_bytes(t.host, S->slots[t.slot].buf, t.bytes, t.stream);
                std::lock_guard<std::mutex> lock(S->m);
                S->slots[t.slot].busy = false;
                S->done.notify_all();
            }
            continue;
        }
        if (S->stop.load()) return;
        // an upload's pieces run out before it closes: look again only for something new
        const int all = S->up.n;
        for (int i = 0; i < kSpins; ++i) {
            if (S->landings.load(std::memory_order_relaxed) > 0 || S->stop.load(std::memory_order_relaxed) ||
                (S->up_open.load(std::memory_order_relaxed) && S->up.next.load(std::memory_order_relaxed) < all))
                break;
            spin_pause();
        }
        if (S->landings.load() > 0 || (S->up_open.load() && S->up.next.load() < S->up.n)) continue;
        mine.asleep.store(true);
        if (work() && mine.asleep.exchange(false)) continue;
        sem_wait(&mine.sem);
    }
}

// The next slot of the ring, free: its previous piece has landed, or its
// previous upload's copy is done.
static cudaError_t take_slot(ppt_stager* S, int* out) {
    const int k = (int)S->next;
    S->next = (S->next + 1) % S->slots.size();
    StagerSlot& slot = S->slots[k];
    cudaError_t e = cudaSuccess;
    if (slot.in_flight) {
        e = cudaEventSynchronize(slot.ev);
        slot.in_flight = false;
    }
    std::unique_lock<std::mutex> lock(S->m);
    S->done.wait(lock, [&] { return !slot.busy; });
    *out = k;
    return e;
}

// Piece size of a copy: every thread gets a share or more, within [kMinPiece, slot].
static int64_t piece_bytes(const ppt_stager* S, int64_t bytes) {
    int64_t p = ((bytes + 2 * S->pool - 1) / (2 * S->pool) + 4095) / 4096 * 4096;
    if (p < kMinPiece) p = kMinPiece;
    return p < S->slot_bytes ? p : S->slot_bytes;
}

// src -> dst in turns of half the ring, so that the copies of one turn cross
// while the next is being staged.
static cudaError_t upload(ppt_stager* S, char* dst, const char* src, int64_t bytes) {
    const int64_t piece = piece_bytes(S, bytes);
    const int64_t turn = piece * (int64_t)(S->slots.size() / 2);
    StagerUpload& U = S->up;
    for (int64_t a = 0; a < bytes; a += turn) {
        const int64_t b = a + turn < bytes ? a + turn : bytes;
        const int n = (int)((b - a + piece - 1) / piece);
        const int first = (int)S->next;
        for (int i = 0; i < n; ++i) {
            int k;
            const cudaError_t e = take_slot(S, &k);
            if (e != cudaSuccess) return e;
        }
        U.dev = dst + a;
        U.host = src + a;
        U.bytes = b - a;
        U.piece = piece;
        U.first = first;
        U.n = n;
        U.stream = bytes > kStreamBytes;
        U.next = 0;
        U.done = 0;
        U.error = 0;
        if (n > 1) {
            S->up_open.store(true);
            const int64_t help = (b - a) / kBytesPerThread;      // and the caller
            wake(S, (int)(help < 1 ? 1 : help));
        }
        claim_pieces(S);
        while (U.done.load() < n) spin_pause();
        if (n > 1) {                          // no thread is at it any more: U and src are the caller's again
            S->up_open.store(false);
            while (S->joined.load() > 0) spin_pause();
        }
        if (U.error.load()) return (cudaError_t)U.error.load();
    }
    return cudaSuccess;
}

static cudaError_t download(ppt_stager* S, char* dst, const char* src, int64_t bytes) {
    const int64_t piece = piece_bytes(S, bytes);
    for (int64_t a = 0; a < bytes; a += piece) {
        const int64_t b = a + piece < bytes ? a + piece : bytes;
        int k;
        cudaError_t e = take_slot(S, &k);
        StagerSlot& slot = S->slots[k];
        if (e == cudaSuccess) e = cudaMemcpyAsync(slot.buf, src + a, (size_t)(b - a), cudaMemcpyDeviceToHost, S->stream);
        if (e == cudaSuccess) e = cudaEventRecord(slot.ev, S->stream);
        if (e != cudaSuccess) return e;
        std::lock_guard<std::mutex> lock(S->m);
        slot.busy = true;
        slot.seq = ++S->queued;
        S->arriving.push(StagerLanding{k, dst + a, b - a, bytes > kStreamBytes, std::this_thread::get_id()});
        S->arrival.notify_one();
    }
    return cudaSuccess;
}

// After an error, with S->ring held: nothing of the call is in flight any more
// (downloads beyond the first `before`, an upload's copies), so the caller may
// give its memory back.
static void settle(ppt_stager* S, uint64_t before) {
    cudaStreamSynchronize(S->stream);
    std::unique_lock<std::mutex> lock(S->m);
    S->done.wait(lock, [&] {
        for (const StagerSlot& s : S->slots)
            if (s.busy && s.seq > before) return false;
        return true;
    });
}

// A caller's handle is a number that no later stager gets, looked up here: a
// handle that has been destroyed is an error (or nothing left to destroy), also for
// an owner that does not know of it.
struct StagerTable {
    std::mutex m;
    std::map<uintptr_t, ppt_stager*> live;
    uintptr_t last = 0;
};
static StagerTable& stagers() {
    static StagerTable* t = new StagerTable;      // outlives the threads of the process's end
    return *t;
}
static ppt_stager* live_stager(ppt_stager* handle) {
    StagerTable& t = stagers();
    std::lock_guard<std::mutex> lock(t.m);
    const auto at = t.live.find(reinterpret_cast<uintptr_t>(handle));
    return at == t.live.end() ? nullptr : at->second;
}

// The stager's device is current while one of its calls runs.
struct OnDevice {
    int prev = 0;
    explicit OnDevice(int device) {
        cudaGetDevice(&prev);
        if (prev != device) cudaSetDevice(device);
        else prev = -1;
    }
    ~OnDevice() {
        if (prev >= 0) cudaSetDevice(prev);
    }
};

static void destroy_stager(ppt_stager* S) {
    // the waiter first: it hands its last arrivals to the pool
    if (!S->threads.empty() && (int)S->threads.size() > S->pool) {
        {
            std::lock_guard<std::mutex> lock(S->m);
            S->stop_waiter = true;
        }
        S->arrival.notify_all();
        S->threads.back().join();
        S->threads.pop_back();
    }
    S->stop.store(true);
    for (int k = 0; k < (int)S->threads.size(); ++k) sem_post(&S->sleepers[k].sem);
    for (std::thread& t : S->threads) t.join();
    {
        OnDevice on(S->device);
        if (S->stream) cudaStreamSynchronize(S->stream);
        for (StagerSlot& s : S->slots)
            if (s.ev) cudaEventDestroy(s.ev);
        if (S->pinned) cudaFreeHost(S->pinned);
    }
    delete S;
}

}  // namespace ppt

using namespace ppt;

extern "C" int ppt_stager_destroy(ppt_stager* handle) {
    ppt_stager* S = nullptr;
    {
        StagerTable& t = stagers();
        std::lock_guard<std::mutex> lock(t.m);
        const auto at = t.live.find(reinterpret_cast<uintptr_t>(handle));
        if (at == t.live.end()) return PPT_OK;
        S = at->second;
        t.live.erase(at);
    }
    destroy_stager(S);
    return PPT_OK;
}

extern "C" int ppt_stager_create(int64_t slot_bytes, int n_slots, int n_threads, void* copy_stream, ppt_stager** out) {
    if (!out) return fail(PPT_ERR_ARG, "out must not be NULL");
    *out = nullptr;
    if (slot_bytes < 4096 || n_slots < 2 || n_threads < 1 || n_slots > 4096 || n_threads > 256)
        return fail(PPT_ERR_ARG, "a stager needs slots of 4096 bytes or more, 2 to 4096 of them and 1 to 256 threads");
    ppt_stager* S = nullptr;
    try {
        S = new ppt_stager;
        S->slots.resize((size_t)n_slots);
        S->arriving.at.resize((size_t)n_slots);
        S->land.at.resize((size_t)n_slots);
        S->slot_bytes = slot_bytes;
        S->stream = static_cast<cudaStream_t>(copy_stream);
        cudaError_t e = cudaGetDevice(&S->device);
        if (e == cudaSuccess) e = cudaHostAlloc(&S->pinned, (size_t)slot_bytes * n_slots, cudaHostAllocDefault);
        for (int k = 0; e == cudaSuccess && k < n_slots; ++k) {
            S->slots[k].buf = S->pinned + (size_t)slot_bytes * k;
            e = cudaEventCreateWithFlags(&S->slots[k].ev, cudaEventDisableTiming);
        }
        if (e != cudaSuccess) {
            destroy_stager(S);
            return e == cudaErrorMemoryAllocation ? fail(PPT_ERR_OOM, "pinned staging buffers") : cuda_fail(e, "stager");
        }
        S->pool = n_threads;
        S->sleepers.reset(new StagerSleeper[n_threads]);
        S->threads.reserve((size_t)n_threads + 1);
        for (int t = 0; t < n_threads; ++t) S->threads.emplace_back(stager_worker, S, t);
        S->threads.emplace_back(stager_waiter, S);
        StagerTable& t = stagers();
        std::lock_guard<std::mutex> lock(t.m);
        t.live.emplace(++t.last, S);
        *out = reinterpret_cast<ppt_stager*>(t.last);
    } catch (const std::exception& ex) {
        if (S) destroy_stager(S);
        return fail(PPT_ERR_OOM, std::string("stager: ") + ex.what());
    }
    return PPT_OK;
}

extern "C" int ppt_stager_upload(ppt_stager* handle, void* dst, const void* src, int64_t bytes, void* stream) {
    ppt_stager* S = live_stager(handle);
    if (!S || bytes < 0 || (bytes > 0 && (!dst || !src))) return fail(PPT_ERR_ARG, "not a stager, or dst or src NULL");
    if (bytes == 0) return PPT_OK;
    try {
        std::lock_guard<std::mutex> ring(S->ring);
        OnDevice on(S->device);
        cudaStream_t user = static_cast<cudaStream_t>(stream);
        cudaEvent_t ev = nullptr;
        // dst may be memory that work queued on the caller's stream still uses
        PPT_CUDA_TRY(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
        cudaError_t e = cudaEventRecord(ev, user);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(S->stream, ev, 0);
        if (e == cudaSuccess) e = upload(S, static_cast<char*>(dst), static_cast<const char*>(src), bytes);
        if (e == cudaSuccess) e = cudaEventRecord(ev, S->stream);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(user, ev, 0);
        if (e != cudaSuccess) cudaStreamSynchronize(S->stream);   // dst may go once the call has failed
        cudaEventDestroy(ev);
        return e == cudaSuccess ? PPT_OK : cuda_fail(e, "staged upload");
    } catch (const std::exception& ex) {
        return fail(PPT_ERR_OOM, std::string("stager: ") + ex.what());
    }
}

extern "C" int ppt_stager_download(ppt_stager* handle, void* dst, const void* src, int64_t bytes, void* after) {
    ppt_stager* S = live_stager(handle);
    if (!S || bytes < 0 || (bytes > 0 && (!dst || !src))) return fail(PPT_ERR_ARG, "not a stager, or dst or src NULL");
    try {
        std::lock_guard<std::mutex> ring(S->ring);
        OnDevice on(S->device);
        const uint64_t before = S->queued;
        cudaError_t e = after ? cudaStreamWaitEvent(S->stream, static_cast<cudaEvent_t>(after), 0) : cudaSuccess;
        if (e == cudaSuccess) e = download(S, static_cast<char*>(dst), static_cast<const char*>(src), bytes);
        if (e != cudaSuccess) settle(S, before);
        return e == cudaSuccess ? PPT_OK : cuda_fail(e, "staged download");
    } catch (const std::exception& ex) {
        return fail(PPT_ERR_OOM, std::string("stager: ") + ex.what());
    }
}

extern "C" int ppt_stager_finish(ppt_stager* handle) {
    ppt_stager* S = live_stager(handle);
    if (!S) return fail(PPT_ERR_ARG, "not a stager");
    try {
        std::unique_lock<std::mutex> lock(S->m);
        const uint64_t upto = S->queued;
        S->done.wait(lock, [&] {
            for (const StagerSlot& s : S->slots)
                if (s.busy && s.seq <= upto) return false;
            return true;
        });
        cudaError_t e = S->lost_error;
        const auto mine = S->errors.find(std::this_thread::get_id());
        if (mine != S->errors.end()) {
            e = mine->second;
            S->errors.erase(mine);
        }
        if (e != cudaSuccess) return cuda_fail(e, "staged copy");
        return PPT_OK;
    } catch (const std::exception& ex) {
        return fail(PPT_ERR_OOM, std::string("stager: ") + ex.what());
    }
}
