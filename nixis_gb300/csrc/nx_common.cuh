// nx_common.cuh -- shared definitions for the nixis_gb300 CUDA library.
#pragma once

#include <cstdint>
#include <cstdio>
#include <cuda_runtime.h>

#include "../../include/nixis_gb300.h"

#define NX_EXPORT extern "C" __attribute__((visibility("default")))

namespace nx {

// Records the message returned by nx_last_error() for this host thread.
void set_error(const char *fmt, ...);
int fail(int code, const char *fmt, ...);
int check_cuda(cudaError_t e, const char *what);

// Number of SMs of the current device (cached per device).
int sm_count();

}  // namespace nx

#define NX_CHECK_CUDA(expr)                                   \
    do {                                                      \
        cudaError_t _e = (expr);                              \
        if (_e != cudaSuccess) return nx::check_cuda(_e, #expr); \
    } while (0)

#define NX_CHECK_LAUNCH(name)                                 \
    do {                                                      \
        cudaError_t _e = cudaGetLastError();                  \
        if (_e != cudaSuccess) return nx::check_cuda(_e, name); \
    } while (0)

// Tile tables (nx_tiling) hold an updatable row's six slots as three 16-byte
// pairs of edges and three words of neighbours, rows in groups of 32, a
// group's three planes one after the other: slot pair x of row l is unit
// tile_unit(l) + 32 x.  A warp's 32 rows of a plane are 512 and 128 bytes in
// one piece, and the planes' addresses differ by constants.
__host__ __device__ __forceinline__ int tile_unit(int l) { return (l >> 5) * 96 + (l & 31); }
