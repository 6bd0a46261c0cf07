// Cases of the stager on the stand-in runtime (ppt_internal.cuh beside this
// file): main <case>, status 0 when it holds.
#include "staging.cu"

#include <chrono>
#include <cstdio>

static void expect(bool ok, const char* what) {
    if (ok) return;
    std::fprintf(stderr, "FAILED: %s\n", what);
    std::_Exit(1);
}

struct Ring {
    FakeStream copy;
    ppt_stager* s = nullptr;
    explicit Ring(int slots = 8, int threads = 3) {
        expect(ppt_stager_create(1 << 20, slots, threads, &copy, &s) == PPT_OK, "create");
    }
    ~Ring() { ppt_stager_destroy(s); }
};

// An event that holds a stream until open().
struct Gate {
    FakeEvent ev;
    Gate() { ev.mark = std::make_shared<FakeMark>(); }
    void open() { ev.mark->complete(0); }
};

// A download refused after some of its pieces were queued: none of them is in
// flight when it returns.
static void refused_download() {
    Ring ring;
    Gate gate;
    std::vector<char> src(3 << 20, 1), dst(3 << 20, 0);
    std::atomic<bool> opened{false};
    std::thread later([&] {
        std::this_thread::sleep_for(std::chrono::milliseconds(100));
        opened = true;
        gate.open();
    });
    fake_copies_left = 2;
    const int rc = ppt_stager_download(ring.s, dst.data(), src.data(), (int64_t)src.size(), &gate.ev);
    const bool settled = opened.load() && fake_in_flight.load() == 0;
    fake_copies_left = 1 << 30;
    later.join();
    expect(rc == PPT_ERR_CUDA, "the download reports the refused copy");
    expect(settled, "its other pieces have landed");
    const std::vector<char> at_return = dst;
    expect(ppt_stager_finish(ring.s) == PPT_OK, "finish");
    expect(dst == at_return, "nothing is written after the return");
    expect(ppt_stager_download(ring.s, dst.data(), src.data(), (int64_t)src.size(), nullptr) == PPT_OK &&
               ppt_stager_finish(ring.s) == PPT_OK && dst == src, "the next download");
}

// An upload refused after some of its copies were queued: the destination is
// free when it returns.
static void refused_upload() {
    Ring ring;
    Gate gate;
    FakeStream user;
    cudaStreamWaitEvent(&user, &gate.ev, 0);
    std::vector<char> src(3 << 20, 1), dst(3 << 20, 0);
    std::thread later([&] {
        std::this_thread::sleep_for(std::chrono::milliseconds(100));
        gate.open();
    });
    fake_copies_left = 2;
    const int rc = ppt_stager_upload(ring.s, dst.data(), src.data(), (int64_t)src.size(), &user);
    const int in_flight = fake_in_flight.load();
    fake_copies_left = 1 << 30;
    later.join();
    expect(rc == PPT_ERR_CUDA, "the upload reports the refused copy");
    expect(in_flight == 0, "its other copies have run");
}

// A download that fails is an error of the thread that queued it, whoever
// finishes first.
static void error_of_its_caller() {
    Ring ring;
    std::vector<char> bad(1000, 1), good(1000, 2), a(1000), b(1000);
    fake_bad_source = bad.data();
    expect(ppt_stager_download(ring.s, a.data(), bad.data(), 1000, nullptr) == PPT_OK, "queue");
    int other = -100;
    std::thread([&] {
        other = ppt_stager_download(ring.s, b.data(), good.data(), 1000, nullptr);
        if (other == PPT_OK) other = ppt_stager_finish(ring.s);
    }).join();
    expect(other == PPT_OK && b == good, "another thread's download is good");
    expect(ppt_stager_finish(ring.s) == PPT_ERR_CUDA, "the failed one is reported to its caller");
    fake_bad_source = nullptr;
    expect(ppt_stager_finish(ring.s) == PPT_OK, "once");
}

// A handle outlives its stager: destroying it again is nothing, using it an error,
// and a later stager does not get it.
static void destroyed_twice() {
    FakeStream copy;
    ppt_stager *first = nullptr, *second = nullptr;
    char a[8] = {}, b[8] = {};
    expect(ppt_stager_create(4096, 2, 1, &copy, &first) == PPT_OK, "create");
    expect(ppt_stager_download(first, a, b, 8, nullptr) == PPT_OK, "a download that nothing waits for");
    expect(ppt_stager_destroy(first) == PPT_OK && ppt_stager_destroy(first) == PPT_OK, "destroy twice");
    expect(ppt_stager_create(4096, 2, 1, &copy, &second) == PPT_OK && second != first, "another one");
    expect(ppt_stager_destroy(first) == PPT_OK && ppt_stager_finish(first) == PPT_ERR_ARG, "the old handle");
    expect(ppt_stager_finish(second) == PPT_OK && ppt_stager_destroy(second) == PPT_OK, "the new one");
}

// Uploads and downloads from several threads: every byte (and, built with
// -fsanitize=thread, no data race).
static void several_callers() {
    Ring ring(8, 3);
    std::atomic<int> wrong{0};
    std::vector<std::thread> callers;
    for (int k = 0; k < 4; ++k)
        callers.emplace_back([&, k] {
            FakeStream user;
            for (int i = 0; i < 8; ++i) {
                const size_t n = (size_t)(k + 1) * 300001 + (size_t)i * 4097;
                std::vector<char> src(n), dev(n), dst(n);
                for (size_t q = 0; q < n; ++q) src[q] = (char)(q * 31 + k + i);
                FakeEvent ev;
                if (ppt_stager_upload(ring.s, dev.data(), src.data(), (int64_t)n, &user)) ++wrong;
                cudaEventRecord(&ev, &user);
                if (ppt_stager_download(ring.s, dst.data(), dev.data(), (int64_t)n, &ev)) ++wrong;
                if (ppt_stager_finish(ring.s) || dst != src) ++wrong;
                cudaStreamSynchronize(&user);
            }
        });
    for (std::thread& t : callers) t.join();
    expect(wrong == 0, "every byte");
}

int main(int argc, char** argv) {
    const std::string which = argc > 1 ? argv[1] : "";
    if (which == "refused_download") refused_download();
    else if (which == "refused_upload") refused_upload();
    else if (which == "error_of_its_caller") error_of_its_caller();
    else if (which == "destroyed_twice") destroyed_twice();
    else if (which == "several_callers") several_callers();
    else return 2;
    return 0;
}
