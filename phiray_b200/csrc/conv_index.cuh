// The weight-stationary convolution's places of a patch vector (nn.cu
// k_conv_ws), worked out once a block; plain arithmetic, so that a host build
// can hold it to every image size.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define CONV_HD __host__ __device__ __forceinline__
#else
#define CONV_HD inline
#endif

namespace phx {

// Vector v of a patch (pixel after pixel, `groups` 8-channel groups each, at most
// 8; rows of `px` pixels): its pixel against the patch's first in an image `W`
// wide, and in one word its group (bits 0-2), its place in shared memory in bytes
// (4-14, a multiple of 16; groups `lbo` bytes apart), row (16-20) and column (24-27).
struct PatchVec {
    uint32_t pixel, word;

    CONV_HD PatchVec() : pixel(0), word(0) {}
    CONV_HD PatchVec(int v, int groups, int px, int lbo, int W) {
        const int g = v % groups, q = v / groups, row = q / px, col = q - row * px;
        word = (uint32_t)(g * lbo + q * 16) | (uint32_t)g | (uint32_t)row << 16 | (uint32_t)col << 24;
        pixel = pixel_in(W);
    }
    // 32 bits hold it for every row of an image that fits the memory; the rows
    // past the image are not used.
    CONV_HD uint32_t pixel_in(int W) const { return (uint32_t)row() * (uint32_t)W + (uint32_t)column(); }
    CONV_HD uint32_t shared_bytes() const { return word & 0x7FF0u; }
    CONV_HD uint32_t channel() const { return (word & 7u) * 8u; }
    CONV_HD int row() const { return (int)((word >> 16) & 31u); }
    CONV_HD int column() const { return (int)(word >> 24); }
};

}  // namespace phx
