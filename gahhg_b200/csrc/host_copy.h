// host_copy.h - host memory copies by several threads.
//
// One thread copies 7-17 GB/s here (a pageable cudaMemcpy is such a copy
// inside the driver), the link to the device takes 52 GB/s: six threads keep
// it busy.
#pragma once
#include <atomic>
#include <condition_variable>
#include <cstdint>
#include <functional>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

#include <cuda_runtime.h>

#include "gahhg.h"

namespace gahhg {

// memcpy to memory that the device reads next, past the caches: copies to the
// device of lines that lie dirty in the cores' caches ran at 13-20 GB/s, of
// lines in memory at 44 (160 MB through the ring below).
void copy_for_device(void* to, const void* from, size_t bytes);

// A fixed set of threads that work through the slices of one job at a time.
class CopyTeam {
public:
    CopyTeam() = default;
    ~CopyTeam();
    CopyTeam(const CopyTeam&) = delete;
    CopyTeam& operator=(const CopyTeam&) = delete;

    // Starts up to `workers` threads; false when none could be started.
    bool start(int workers) noexcept;
    bool running() const { return !threads.empty(); }
    // The workers a machine of this size is given (0: too small to gain).
    static int default_workers();

    // Begins a job: work(i) for i in [0, n), slices below `limit` at once, the
    // others as allow() raises it.  Jobs follow one another: every post() is
    // answered by one finish().
    void post(size_t n, size_t limit, std::function<void(size_t)> work);
    void allow(size_t limit) { lim.store(limit, std::memory_order_release); }
    bool done(size_t i) const { return flags[i].load(std::memory_order_acquire) != 0; }
    bool help();            // the caller does one slice; false when none is left
    void finish(bool abort);  // waits for the workers; abort: slices not begun are dropped

private:
    void run();
    bool one(size_t i);
    std::vector<std::thread> threads;
    std::mutex mu;
    std::condition_variable cv, cv_idle;
    uint64_t job = 0;
    int inside = 0;
    bool open = false, stop = false;
    std::function<void(size_t)> fn;
    size_t count = 0, cap = 0;
    std::unique_ptr<std::atomic<uint8_t>[]> flags;
    std::atomic<size_t> next{0}, lim{0};
    std::atomic<bool> dropped{false};
};

// Pageable host memory <-> device through a ring of page-locked slots that a
// team fills or empties while the copies of other slots run.  There is one per
// process, made by the first call that needs it and given back when the last
// grid goes, unless it was in use within KEEP_SECONDS before (programs that
// build, ask and drop one index after another would allocate it each time).  A
// query that finds it in use, or host memory that is page-locked already, is
// copied directly.
class HostStage {
public:
    // 6 MB page-locked (3.7 ms to allocate).  48 MB to the device in 1.15 ms
    // (2.6-3.4 directly); slots of 256 KB 1.4, of 1 MB 1.1 but 16 MB in all.
    static constexpr size_t SLOT = 512 << 10;
    static constexpr size_t SLOTS = 12;
    // 4 MB take 130 us this way and 210 directly; what is smaller gains less
    // than waking the threads costs.
    static constexpr size_t MIN_BYTES = 4 << 20;

    // The process's stage for the calling thread, or null; with `wait` a call
    // that finds it in use waits for its turn.
    static HostStage* acquire(int device, const void* host, size_t bytes, bool wait = false);
    static bool pageable(const void* host);
    static void release(HostStage* s);
    static constexpr double KEEP_SECONDS = 2.0;
    static void grid_made();
    static void grid_gone();

    // Enqueued on `s` when it returns; the host memory has been read.  The
    // second form: arrays that lie one behind the other on the device.
    struct Part {
        const void* host;
        size_t bytes;
    };
    cudaError_t to_device(void* d, const void* h, size_t bytes, cudaStream_t s);
    cudaError_t to_device(void* d, const std::vector<Part>& parts, cudaStream_t s);
    // `h` has been written when it returns.
    cudaError_t to_host(void* h, const void* d, size_t bytes, cudaStream_t s);
    ~HostStage();

private:
    bool create();
    cudaError_t fill(void* d, size_t bytes, cudaStream_t s, const std::function<void(size_t, uint8_t*, size_t)>& read);
    cudaError_t settle();  // the ring's last copies have ended
    CopyTeam team;
    uint8_t* ring = nullptr;
    cudaEvent_t ev[SLOTS] = {};
    int device = -1;
    double used = 0.0;
    int last = -1;  // event of the last copy enqueued
};

}  // namespace gahhg
