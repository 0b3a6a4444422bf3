// Host build of gahhg_b200/csrc/scan_state.cpp with an allocator that fails
// when told to, for tests/test_cpu_scan_state.py (no GPU, no CUDA runtime).
#include "../../gahhg_b200/csrc/scan_state.cpp"

#include <cstdarg>
#include <cstdlib>
#include <cstring>

static int g_calls, g_fail, g_live;

extern "C" {
cudaError_t cudaGetDevice(int* d)
{
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t)
{
    if (++g_calls == g_fail) return cudaErrorUnknown;
    memset(p, v, n);
    return cudaSuccess;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t)
{
    g_live--;
    free(p);
    return cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t) { return "made to fail"; }
}

namespace gahhg {
void set_error(const char*, ...) {}
gahhg_status pool_alloc(void** p, size_t bytes, int, cudaStream_t)
{
    if (++g_calls == g_fail) return GAHHG_ERR_NOMEM;
    *p = malloc(bytes);
    memset(*p, 0xAB, bytes);
    g_live++;
    return GAHHG_OK;
}
}  // namespace gahhg

// Reserves for n1 and then n2 items, the `fail`th allocation or clearing
// failing; after a failure the reserve is asked for once more, and has to
// leave a state that scans can use.  Returns how many of the two failed, or
// -1 with what was wrong in *what.
extern "C" int reserve_with_failure(long n1, long n2, int fail, int* what)
{
    using namespace gahhg;
    g_calls = 0;
    g_fail = fail;
    g_live = 0;
    void* state = nullptr;
    int failed = 0;
    const long n[2] = {n1, n2};
    for (int k = 0; k < 2; k++) {
        gahhg_status r = scan_state_reserve(&state, (size_t)n[k], nullptr);
        if (r != GAHHG_OK) {
            failed++;
            r = scan_state_reserve(&state, (size_t)n[k], nullptr);
        }
        const ScanState* st = (const ScanState*)state;
        const size_t tiles = ((size_t)n[k] + SCAN_TILE - 1) / SCAN_TILE;
        *what = r != GAHHG_OK ? 1 : !st ? 2 : !st->counter ? 3 : *st->counter != 0 ? 4 : !st->status ? 5
                : st->max_tiles < tiles ? 6 : 0;
        for (size_t t = 0; !*what && t < st->max_tiles; t++)
            if (st->status[t]) *what = 7;
        if (*what) return -1;
    }
    scan_state_destroy(state);
    *what = g_live ? 8 : 0;
    return g_live ? -1 : failed;
}
