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

// Whether a convolution of that many images and pixels, F filters and K products per output is for the per-tap kernel: one thread per pixel and four
// filters, one chain of K steps each, and a second launch for bias and activation (`follow`).  The blocked kernels compute whole tiles of 32 or 64 filters, and a launch of theirs takes about
// 8 us however little it has to do (ks as in ln_conv_f32_slice).
//   - little work: 32 filters of 1x1 over one channel, 64 x 64 pixels: 4.2 us against 12.4; 16 of 3x3 over one: 6.2 / 8.4; 32 over four (K = 36): 12.4 /
//     16.5, over eight (K = 72): 18.5 / 14.5; two filters over four: 12.4 / 10.3
//   - few filters of a general kernel, which pays for finding every tap: one 5x5 filter over eight channels, 256 x 256: 23 / 66 us, four of them
//     43 / 66, eight 70 / 68; 64 x 64 pixels: 21 / 21, 35 / 21; one over four
//     channels, 32 x 32 (K = 100): 12 / 21
//   - a single 3x3 filter on a large image: 16 channels, 512 x 512: 66 / 93 us, 256 x 256: 27 / 31; two filters: 117 / 94
// Up to 63 products neither kernel splits a sum and both add in the same order, so the batch may decide; beyond, one image does.
inline bool ln_conv_f32_per_tap(int64_t images, int64_t plane, int64_t F, int64_t K, int ks, bool follow) {
    if (!follow && K <= 36 && (ks == 0 || 4 * F >= K) && images * plane * ((F + 3) / 4) <= 65536) return true;
    const int64_t pixels = K < 64 ? images * plane : plane;
    if (ks == 0) return (F <= (K < 64 ? 8 : 4) && pixels >= 8192 * F) || (F == 1 && K <= 128);
    return F == 1 && (ks == 3 || K == 1) && pixels >= 65536;
}

// Slice of the k range that a kernel holds in shared memory: four channels of a 3x3 kernel or 32 of a 1x1 one where operands are copied
// asynchronously (`async`), else one channel, or eight k of any other kernel (ks = 1: 1x1 without padding, 3: 3x3 without dilation, 0: anything).
constexpr int ln_conv_f32_slice(bool async, int ks) { return async ? (ks == 3 ? 36 : 32) : (ks == 3 ? 9 : 8); }

// Part z of a k range of `slices` slices cut into `parts` begins with this one: whole slices, as evenly as they go.
constexpr int ln_conv_f32_first_slice(int slices, int z, int parts) { return slices * z / parts; }  // (at most 2^21 slices)

struct ln_conv_f32_cut {
    int bm, bn, parts;  // filters and pixels of a tile; CTAs of the cluster over which a tile's k range is split
};

// Ungrouped convolution with optional bias and activation.  Tile: 64 filters x 128 pixels while that gives every SM four CTAs (of four
// warps) even without splitting, 64 x 64 below; layers of at most 32 filters 32 x 128.  The k range is split over clusters of up to eight
// CTAs until a single image has about eight CTAs of two warps per SM of a B200, in parts of at least two slices (four of the short ones of
// operands staged through registers).  The split looks at one image and not at the batch: it is what the order of a sum depends on, and an
// image has the same outputs in any batch.
// one_chain: no split, so that every output is one chain of fused multiply-adds.  Calibration asks for it: the scales of an 8-bit
// network, and with them its codes, must not depend on how the work was cut.
inline ln_conv_f32_cut ln_conv_f32_choose(int sm_count, int64_t images, int64_t plane, int64_t F, int64_t K, int ks, bool async, bool one_chain) {
    const bool narrow = !async && F <= 32;
    auto tiles = [&](int64_t pixels, int bm, int bn) { return ((pixels + bn - 1) / bn) * ((F + bm - 1) / bm); };
    auto wide = [&](int64_t pixels, int sms) { return async && ((pixels + 127) / 128 * 128 - pixels) * 10 <= pixels && tiles(pixels, 64, 128) * 8 >= 2ll * sms; };
    ln_conv_f32_cut c;
    c.bm = narrow ? 32 : 64;
    c.bn = narrow || wide(images * plane, sm_count) ? 128 : 64;
    constexpr int kSms = 148;
    const bool wide1 = wide(plane, kSms);
    const int64_t tiles1 = tiles(plane, c.bm, narrow || wide1 ? 128 : 64), most = (wide1 ? 4ll : 8ll) * kSms;
    c.parts = 1;
    while (!one_chain && c.parts < 8 && tiles1 * c.parts * 2 <= most && K / (c.parts * 2) >= (async ? 2 : 4) * ln_conv_f32_slice(async, ks)) c.parts *= 2;
    return c;
}
