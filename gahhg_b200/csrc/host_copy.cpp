// host_copy.cpp - see host_copy.h.
#include "host_copy.h"

#include <algorithm>
#include <chrono>
#include <cstring>
#include <new>

#if defined(__SSE2__)
#include <emmintrin.h>
#endif

namespace gahhg {

namespace {

double now_seconds()
{
    return std::chrono::duration<double>(std::chrono::steady_clock::now().time_since_epoch()).count();
}

}  // namespace

void copy_for_device(void* to, const void* from, size_t bytes)
{
#if defined(__SSE2__)
    if (((uintptr_t)to & 15u) == 0) {
        __m128i* d = (__m128i*)to;
        const __m128i* s = (const __m128i*)from;
        const size_t lines = bytes / 64;
        for (size_t i = 0; i < lines; i++, d += 4, s += 4) {
            const __m128i a = _mm_loadu_si128(s), b = _mm_loadu_si128(s + 1);
            const __m128i c = _mm_loadu_si128(s + 2), e = _mm_loadu_si128(s + 3);
            _mm_stream_si128(d, a);
            _mm_stream_si128(d + 1, b);
            _mm_stream_si128(d + 2, c);
            _mm_stream_si128(d + 3, e);
        }
        _mm_sfence();
        to = d;
        from = s;
        bytes %= 64;
    }
#endif
    memcpy(to, from, bytes);
}

int CopyTeam::default_workers()
{
    const int hw = (int)std::thread::hardware_concurrency();
    return hw < 4 ? 0 : std::min(6, hw / 2);
}

bool CopyTeam::start(int workers) noexcept
{
    try {
        threads.reserve((size_t)std::max(workers, 0));
        for (int k = 0; k < workers; k++) threads.emplace_back([this] { run(); });
    } catch (...) {
        // as many as there are
    }
    return running();
}

CopyTeam::~CopyTeam()
{
    {
        std::lock_guard<std::mutex> lk(mu);
        stop = true;
    }
    cv.notify_all();
    for (std::thread& t : threads) t.join();
}

// Slice i, when it is below the limit; waits for that (the poster raises the
// limit or drops the job).
bool CopyTeam::one(size_t i)
{
    while (i >= lim.load(std::memory_order_acquire)) {
        if (dropped.load(std::memory_order_acquire)) return false;
        std::this_thread::yield();
    }
    if (dropped.load(std::memory_order_acquire)) return false;
    fn(i);
    flags[i].store(1, std::memory_order_release);
    return true;
}

void CopyTeam::run()
{
    uint64_t seen = 0;
    std::unique_lock<std::mutex> lk(mu);
    for (;;) {
        cv.wait(lk, [&] { return stop || (open && job != seen); });
        if (stop) return;
        seen = job;
        inside++;
        lk.unlock();
        for (;;) {
            const size_t i = next.fetch_add(1, std::memory_order_relaxed);
            if (i >= count || !one(i)) break;
        }
        lk.lock();
        if (--inside == 0) cv_idle.notify_all();
    }
}

void CopyTeam::post(size_t n, size_t limit, std::function<void(size_t)> work)
{
    {
        std::lock_guard<std::mutex> lk(mu);  // no worker is inside: finish() waited for them
        if (n > cap) {
            flags.reset(new std::atomic<uint8_t>[n]);
            cap = n;
        }
        for (size_t i = 0; i < n; i++) flags[i].store(0, std::memory_order_relaxed);
        fn = std::move(work);
        count = n;
        next.store(0, std::memory_order_relaxed);
        lim.store(limit, std::memory_order_relaxed);
        dropped.store(false, std::memory_order_relaxed);
        open = true;
        job++;
    }
    cv.notify_all();
}

bool CopyTeam::help()
{
    size_t i = next.load(std::memory_order_relaxed);
    while (i < count && i < lim.load(std::memory_order_acquire))
        if (next.compare_exchange_weak(i, i + 1, std::memory_order_relaxed)) return one(i);
    return false;
}

void CopyTeam::finish(bool abort)
{
    if (abort) dropped.store(true, std::memory_order_release);
    std::unique_lock<std::mutex> lk(mu);
    open = false;  // a worker that was not woken yet stays out of this job
    cv_idle.wait(lk, [&] { return inside == 0; });
    lk.unlock();
    // slices nobody took, when no worker woke in time
    if (!abort)
        while (help()) {
        }
}

// ---------------------------------------------------------------- stage --

namespace {
std::mutex g_stage_mu;
std::condition_variable g_stage_cv;
HostStage* g_stage = nullptr;  // never destroyed at exit: its threads may outlive static objects
bool g_stage_busy = false;
long long g_grids = 0;
}  // namespace

bool HostStage::create()
{
    if (!team.start(CopyTeam::default_workers())) return false;
    if (cudaHostAlloc((void**)&ring, SLOT * SLOTS, cudaHostAllocPortable) != cudaSuccess) {
        cudaGetLastError();
        ring = nullptr;
        return false;
    }
    return true;
}

HostStage::~HostStage()
{
    for (cudaEvent_t e : ev)
        if (e) cudaEventDestroy(e);
    if (ring) cudaFreeHost(ring);
    cudaGetLastError();
}

bool HostStage::pageable(const void* host)
{
    cudaPointerAttributes at{};
    if (cudaPointerGetAttributes(&at, host) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return at.type == cudaMemoryTypeUnregistered;
}

HostStage* HostStage::acquire(int dev, const void* host, size_t bytes, bool wait)
{
    if (bytes < MIN_BYTES || CopyTeam::default_workers() == 0) return nullptr;
    if (!pageable(host)) return nullptr;
    std::unique_lock<std::mutex> lk(g_stage_mu);
    if (g_stage_busy && !wait) return nullptr;
    g_stage_cv.wait(lk, [] { return !g_stage_busy; });
    if (!g_stage) {
        HostStage* s = new (std::nothrow) HostStage();
        if (!s) return nullptr;
        if (!s->create()) {
            delete s;
            return nullptr;
        }
        g_stage = s;
    }
    HostStage* s = g_stage;
    if (s->device != dev) {  // events belong to a device
        for (cudaEvent_t& e : s->ev) {
            if (e) cudaEventDestroy(e);
            e = nullptr;
        }
        s->last = -1;
        s->device = -1;
        for (cudaEvent_t& e : s->ev)
            if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
                cudaGetLastError();
                return nullptr;
            }
        s->device = dev;
    }
    g_stage_busy = true;
    return s;
}

void HostStage::release(HostStage* s)
{
    if (!s) return;
    s->settle();  // the next user writes the ring, maybe from another device
    {
        std::lock_guard<std::mutex> lk(g_stage_mu);
        g_stage_busy = false;
        s->used = now_seconds();
    }
    g_stage_cv.notify_one();
}

void HostStage::grid_made()
{
    std::lock_guard<std::mutex> lk(g_stage_mu);
    g_grids++;
}

void HostStage::grid_gone()
{
    HostStage* gone = nullptr;
    {
        std::lock_guard<std::mutex> lk(g_stage_mu);
        if (--g_grids == 0 && !g_stage_busy && g_stage && now_seconds() - g_stage->used > KEEP_SECONDS)
            std::swap(gone, g_stage);
    }
    delete gone;
}

cudaError_t HostStage::settle()
{
    if (last < 0) return cudaSuccess;
    const cudaError_t e = cudaEventSynchronize(ev[last]);
    last = -1;
    return e;
}

cudaError_t HostStage::to_device(void* d, const void* h, size_t bytes, cudaStream_t s)
{
    return fill(d, bytes, s, [h](size_t from, uint8_t* to, size_t n) { copy_for_device(to, (const uint8_t*)h + from, n); });
}

cudaError_t HostStage::to_device(void* d, const std::vector<Part>& parts, cudaStream_t s)
{
    std::vector<size_t> end(parts.size());
    size_t bytes = 0;
    for (size_t i = 0; i < parts.size(); i++) end[i] = bytes += parts[i].bytes;
    return fill(d, bytes, s, [&](size_t from, uint8_t* to, size_t n) {
        size_t k = std::upper_bound(end.begin(), end.end(), from) - end.begin();
        while (n > 0) {
            const size_t at = from - (end[k] - parts[k].bytes), m = std::min(n, parts[k].bytes - at);
            copy_for_device(to, (const uint8_t*)parts[k].host + at, m);
            from += m;
            to += m;
            n -= m;
            k++;
        }
    });
}

// read(from, to, n): bytes [from, from + n) of the source
cudaError_t HostStage::fill(void* d, size_t bytes, cudaStream_t s,
                            const std::function<void(size_t, uint8_t*, size_t)>& read)
{
    cudaError_t e = settle();
    if (e != cudaSuccess || bytes == 0) return e;
    const size_t n = (bytes + SLOT - 1) / SLOT;
    const auto end_of = [&](size_t i) { return std::min(bytes, i * SLOT); };
    team.post(n, SLOTS, [=, &read](size_t i) {
        read(i * SLOT, ring + (i % SLOTS) * SLOT, std::min(SLOT, bytes - i * SLOT));
    });
    size_t sent = 0, freed = 0;        // slices enqueued; slices whose copies have ended
    size_t run_end[SLOTS];             // by event: the end of the run it follows
    size_t run_head = 0, run_tail = 0; // runs in flight, oldest first: event run % SLOTS
    while (sent < n && e == cudaSuccess) {
        size_t to = sent;
        const size_t wrap = sent - sent % SLOTS + SLOTS;  // a run is contiguous in the ring
        while (to < n && to < wrap && team.done(to)) to++;
        if (to > sent && run_tail - run_head < SLOTS) {
            e = cudaMemcpyAsync((uint8_t*)d + sent * SLOT, ring + (sent % SLOTS) * SLOT, end_of(to) - sent * SLOT,
                                cudaMemcpyHostToDevice, s);
            const int k = (int)(run_tail % SLOTS);
            if (e == cudaSuccess) e = cudaEventRecord(ev[k], s);
            if (e != cudaSuccess) break;
            last = k;
            run_end[k] = to;
            run_tail++;
            sent = to;
        }
        if (run_head < run_tail) {
            const cudaError_t q = cudaEventQuery(ev[run_head % SLOTS]);
            if (q == cudaSuccess) {
                freed = run_end[run_head % SLOTS];
                run_head++;
                team.allow(freed + SLOTS);
            } else if (q != cudaErrorNotReady) {
                e = q;
            }
        } else if (to == sent) {
            std::this_thread::yield();
        }
    }
    team.finish(e != cudaSuccess);
    if (e != cudaSuccess) cudaGetLastError();
    return e;
}

cudaError_t HostStage::to_host(void* h, const void* d, size_t bytes, cudaStream_t s)
{
    cudaError_t e = settle();
    if (e != cudaSuccess || bytes == 0) return e;
    const size_t n = (bytes + SLOT - 1) / SLOT;
    const auto end_of = [&](size_t i) { return std::min(bytes, i * SLOT); };
    team.post(n, 0, [=](size_t i) {
        memcpy((uint8_t*)h + i * SLOT, ring + (i % SLOTS) * SLOT, std::min(SLOT, bytes - i * SLOT));
    });
    size_t sent = 0, freed = 0;  // slices enqueued; slices copied out
    size_t run_end[SLOTS];
    size_t run_head = 0, run_tail = 0;
    while (freed < n && e == cudaSuccess) {
        const size_t to = std::min({n, freed + SLOTS, sent - sent % SLOTS + SLOTS, sent + SLOTS / 4});
        if (sent < to && run_tail - run_head < SLOTS) {
            e = cudaMemcpyAsync(ring + (sent % SLOTS) * SLOT, (const uint8_t*)d + sent * SLOT, end_of(to) - sent * SLOT,
                                cudaMemcpyDeviceToHost, s);
            const int k = (int)(run_tail % SLOTS);
            if (e == cudaSuccess) e = cudaEventRecord(ev[k], s);
            if (e != cudaSuccess) break;
            last = k;
            run_end[k] = to;
            run_tail++;
            sent = to;
        }
        if (run_head < run_tail) {
            const cudaError_t q = cudaEventQuery(ev[run_head % SLOTS]);
            if (q == cudaSuccess) {
                team.allow(run_end[run_head % SLOTS]);
                run_head++;
            } else if (q != cudaErrorNotReady) {
                e = q;
            }
        } else {
            std::this_thread::yield();
        }
        while (freed < n && team.done(freed)) freed++;
    }
    team.finish(e != cudaSuccess);
    if (e != cudaSuccess) cudaGetLastError();
    return e;
}

}  // namespace gahhg
