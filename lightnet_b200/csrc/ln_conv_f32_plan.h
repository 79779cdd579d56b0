// Host-side rules of the f32 convolution (ln_f32_ops.cu), in plain C++.
#pragma once
#include <cstdint>

// Whether the index arithmetic of the blocked kernels covers an ungrouped convolution of n images, c channels, h x w, into f filters, oh x ow with a
// k x k kernel.  They number pixels (n oh ow), positions in a plane (h w) and the k range (c k^2, times the 64 filters of a tile) in 32 bits, and
// tiles of 64 filters are the y extent of the grid, which ends at 65535.  What they cannot number goes to the per-tap kernel, whose
// offsets have 64 bits and whose threads stride over the outputs.
inline bool ln_conv_f32_blocked(int64_t n, int64_t c, int64_t h, int64_t w, int64_t f, int64_t k, int64_t oh, int64_t ow) {
    return n * oh * ow < (1ll << 30) && h * w < (1ll << 31) && n * c * h * w < (1ll << 40) && c * k * k < (1ll << 24) && (f + 63) / 64 <= 65535;
}
