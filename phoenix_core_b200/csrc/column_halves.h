// How the two halves of an epilogue's warps share the columns of a tile. Plain C++, so that it can be checked without a GPU.
#pragma once

#ifndef PCB_HOST_DEVICE
#ifdef __CUDACC__
#define PCB_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define PCB_HOST_DEVICE inline
#endif
#endif

namespace pcb {

// Columns of the first half of the warps in a tile of `cols` (up to 256), the others' are those behind them: a multiple of the 32 that a warp drains at a
// time, so that no column is stored by both (tiles of 96 and 112 columns cut in the middle had a sixth and a fourteenth of them stored twice).
PCB_HOST_DEVICE int columns_per_half(int cols) { return cols > 128 ? 128 : 64; }

}  // namespace pcb
