// host_copy.h — fills a pinned buffer from many arrays with several threads
// (host code alone, no CUDA: tests/host_copy_host.cpp compiles it for the CPU).
#pragma once

#include <algorithm>
#include <atomic>
#include <cstddef>
#include <cstring>
#include <thread>
#include <vector>

namespace sphrt {

// A part of an array to copy into the pinned buffer.
struct CopyTask {
    const char *src;
    size_t dst, bytes;
};
constexpr size_t TASK_BYTES = 256 << 10;     // largest task
constexpr size_t THREAD_BYTES = 2 << 20;     // input bytes per copying thread (~150 us; creating one takes ~15)
constexpr size_t SEGMENT_BYTES = 8 << 20;    // bytes per copy to the device (~40 us)
constexpr int MAX_COPY_THREADS = 8;

// Copying threads beside the caller for this many bytes.
inline int extra_copy_threads(size_t bytes) {
    const int cores = (int)std::thread::hardware_concurrency();
    return std::min<int>(std::min(MAX_COPY_THREADS, cores / 2) - 1, (int)(bytes / THREAD_BYTES) - 1);
}

// Runs the tasks (ascending dst) into the buffer h of `total` bytes with up to
// `extra` more threads and calls send(from, to) for its segments in order,
// each as soon as its tasks are done.  Where no thread can be had, this one
// does their share.
template <class Send>
void run_copies(char *h, const std::vector<CopyTask> &tasks, size_t total, int extra, Send send) {
    if (extra < 1 || tasks.empty()) {
        for (const CopyTask &t : tasks) std::memcpy(h + t.dst, t.src, t.bytes);
        send((size_t)0, total);
        return;
    }
    const int n = (int)tasks.size();
    // segment k: the tasks up to seg_task[k], the bytes up to seg_end[k]
    std::vector<int> seg_task, seg_of(n);
    std::vector<size_t> seg_end;
    size_t from = 0;
    for (int k = 0; k < n; ++k) {
        const size_t next = k + 1 < n ? tasks[k + 1].dst / 256 * 256 : total;
        seg_of[k] = (int)seg_task.size();
        if (next - from >= SEGMENT_BYTES || k + 1 == n) {
            // a 256-byte boundary at or before the next task: bytes of this one
            // beyond it go with the next segment, which is copied later
            seg_task.push_back(k + 1);
            seg_end.push_back(next);
            from = next;
        }
    }
    const int n_seg = (int)seg_task.size();
    std::vector<std::atomic<int>> left(n_seg);
    for (int g = 0; g < n_seg; ++g) left[g].store(seg_task[g] - (g ? seg_task[g - 1] : 0), std::memory_order_relaxed);
    std::atomic<int> next_task{0};
    auto one = [&]() {
        const int k = next_task.fetch_add(1, std::memory_order_relaxed);
        if (k >= n) return false;
        std::memcpy(h + tasks[k].dst, tasks[k].src, tasks[k].bytes);
        left[seg_of[k]].fetch_sub(1, std::memory_order_release);
        return true;
    };
    std::vector<std::thread> threads;
    try {
        threads.reserve(extra);
        for (int t = 0; t < extra; ++t) threads.emplace_back([&]() { while (one()) {} });
    } catch (...) {
        // no thread or no memory for one: the threads that run, and the loop
        // below, do the rest (they must be joined, so nothing leaves here)
    }
    int seg = 0;
    bool more = true;
    while (seg < n_seg) {
        if (more)
            more = one();
        else
            std::this_thread::yield();
        while (seg < n_seg && left[seg].load(std::memory_order_acquire) == 0) {
            send(seg ? seg_end[seg - 1] : 0, seg_end[seg]);
            ++seg;
        }
    }
    for (std::thread &t : threads) t.join();
}

}  // namespace sphrt
