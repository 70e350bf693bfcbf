// tcr_fold_span.cuh -- the part of a row that lies in a tile of the streamed fold.
//
// Free of CUDA, so that the arithmetic also compiles for the host: positions are 64-bit (an index that needs no
// sort may hold 2^31 elements and more), offsets in a tile 32-bit, and the clamp to the tile comes before the
// narrowing.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define TCR_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define TCR_HOST_DEVICE inline
#endif

namespace tcr {

// Position p relative to the tile [t0, t0 + len), clamped into [0, len].
TCR_HOST_DEVICE int tile_offset(int64_t p, int64_t t0, int len) {
    const int64_t d = p - t0;
    return d <= 0 ? 0 : (d < len ? (int)d : len);
}

}  // namespace tcr
