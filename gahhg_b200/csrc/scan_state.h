// scan_state.h - what the look-back scans (scan.cu) keep between calls.
#pragma once
#include "gahhg_internal.h"

namespace gahhg {

constexpr int SCAN_THREADS = 256;
constexpr int SCAN_ITEMS = 8;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;

struct ScanState {
    unsigned long long* status;
    unsigned int* counter;
    cudaStream_t stream;
    size_t max_tiles;  // tiles `status` holds (0: it is not ready)
    unsigned int tile_base;
    unsigned int epoch;
};

}  // namespace gahhg
