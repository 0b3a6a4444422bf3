// scan_state.cpp - the scans' status words and tile counter.
//
// They come from the library's pool, ordered on the stream that the scans run
// on (cudaMalloc and cudaFree took 100 us each, and a batch or a hierarchy
// build makes a state).  A call that fails leaves no state, or one whose
// status words the next call makes: a state always has its counter.
#include "scan_state.h"

namespace gahhg {

void scan_state_destroy(void* state)
{
    ScanState* st = (ScanState*)state;
    if (!st) return;
    if (st->status) cudaFreeAsync(st->status, st->stream);
    cudaFreeAsync(st->counter, st->stream);
    delete st;
}

// *p = bytes of zeros, or null.
static gahhg_status alloc_cleared(void** p, size_t bytes, int device, cudaStream_t s)
{
    const gahhg_status r = pool_alloc(p, bytes, device, s);
    if (r != GAHHG_OK) {
        *p = nullptr;
        return r;
    }
    const cudaError_t e = cudaMemsetAsync(*p, 0, bytes, s);
    if (e != cudaSuccess) {
        cudaFreeAsync(*p, s);
        *p = nullptr;
    }
    GAHHG_CUDA_TRY(e);
    return GAHHG_OK;
}

gahhg_status scan_state_reserve(void** state, size_t max_n, cudaStream_t s)
{
    const size_t need = (max_n + SCAN_TILE - 1) / SCAN_TILE + 1;
    ScanState* st = (ScanState*)*state;
    if (st && st->max_tiles >= need) return GAHHG_OK;
    int dev = 0;
    GAHHG_CUDA_TRY(cudaGetDevice(&dev));
    if (!st) {
        unsigned int* counter = nullptr;
        GAHHG_TRY(alloc_cleared((void**)&counter, sizeof(unsigned int), dev, s));
        *state = st = new ScanState{nullptr, counter, s, 0, 0, 1};
    }
    // growing: the new array starts cleared and the epoch sequence continues
    if (st->status) cudaFreeAsync(st->status, s);
    st->max_tiles = 0;
    GAHHG_TRY(alloc_cleared((void**)&st->status, 2 * need * sizeof(unsigned long long), dev, s));
    st->max_tiles = 2 * need;
    return GAHHG_OK;
}

}  // namespace gahhg
