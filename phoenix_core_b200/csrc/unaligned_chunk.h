// 16-byte chunks that start at any 16-bit element, read as the aligned vectors of four elements around them. Plain C++, so that the
// bounds can be checked without a GPU.
#pragma once

#ifdef __CUDACC__
#define PCB_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define PCB_HOST_DEVICE inline
#endif

namespace pcb {

// Vectors (1 .. 3), from the aligned one that holds element `at` on, that a chunk of eight elements at `at` reads in a tensor of `total`
// elements (a multiple of 4, up to 2^31 - 4): the third one only if the chunk is not aligned, and none past the end of the tensor.
PCB_HOST_DEVICE int chunk_vectors(int at, int total) {
    const int left = total - (at & ~3);            // at least 4
    return 1 + (left > 4 ? 1 : 0) + ((at & 3) != 0 && left > 8 ? 1 : 0);
}

}  // namespace pcb
