// CPU check of csrc/host_copy.h (run by tests/test_host_copy.py): every byte
// arrives, the segments cover the buffer once and in order, each is complete
// when it is sent, with memory running out after a given number of
// allocations while the threads are made.
#include "../research_codes_gb300/csrc/host_copy.h"

#include <cstdio>
#include <cstdlib>
#include <new>
#include <random>

static std::atomic<long> g_left{-1};   // allocations until the failing ones (-1: none fail)

void *operator new(size_t n) {
    if (g_left.load() >= 0 && g_left.fetch_sub(1) <= 0) {
        g_left.store(0);
        throw std::bad_alloc();
    }
    if (void *p = std::malloc(n ? n : 1)) return p;
    throw std::bad_alloc();
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, size_t) noexcept { std::free(p); }

int main(int argc, char **argv) {
    const int extra = std::atoi(argv[1]);
    const long fail_after = std::atol(argv[2]);   // allocations that succeed once the threads are being made
    const size_t megabytes = (size_t)std::atol(argv[3]);
    (void)argc;
    std::mt19937 rng(7);
    std::vector<sphrt::CopyTask> tasks;
    std::vector<char> src(megabytes << 20);
    for (size_t k = 0; k < src.size(); ++k) src[k] = (char)(k * 2654435761u >> 13);
    size_t o = 0, dst = 1280;   // a header before the first task
    while (o < src.size()) {
        const size_t b = std::min(src.size() - o, (size_t)(1 + rng() % sphrt::TASK_BYTES));
        tasks.push_back(sphrt::CopyTask{src.data() + o, dst, b});
        o += b;
        dst += b;
    }
    const size_t total = (dst + 255) / 256 * 256;
    std::vector<char> h(total, 0), got(total, 0);
    size_t sent = 0;
    bool ordered = true;
    // a first run, as in a process that has copied before; its allocations up
    // to the threads are the next one's
    sphrt::run_copies(h.data(), tasks, total, extra, [&](size_t, size_t) {});
    std::fill(h.begin(), h.end(), 0);
    g_left.store(fail_after < 0 ? -1 : fail_after);
    try {
        sphrt::run_copies(h.data(), tasks, total, extra, [&](size_t from, size_t to) {
            ordered = ordered && from == sent && to >= from && to <= total;
            std::memcpy(got.data() + from, h.data() + from, to - from);
            sent = to;
        });
    } catch (const std::bad_alloc &) {   // before the first thread: the caller's to handle
        g_left.store(-1);
        std::puts("no memory");
        return 0;
    }
    g_left.store(-1);
    for (const sphrt::CopyTask &t : tasks)
        if (std::memcmp(got.data() + t.dst, t.src, t.bytes)) {
            std::puts("bytes differ");
            return 1;
        }
    std::puts(ordered && sent == total ? "ok" : "segments differ");
    return ordered && sent == total ? 0 : 1;
}
