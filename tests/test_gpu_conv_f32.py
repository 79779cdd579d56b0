"""f32 convolution at the edges of its tiles: every output must lie within the rounding bound of a binary32 sum of its products."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def be():
    import lightnet_b200 as ln
    b = ln.B200Backend(0)
    yield b
    b.close()


# batch, channels, height, width, filters, kernel, stride, padding, dilation
@pytest.mark.parametrize("geom", [
    (1, 5, 161, 159, 129, 3, 1, 1, 1),   # k range not a multiple of 4
    (1, 32, 160, 160, 256, 1, 1, 0, 1),  # 64 x 128 tiles, whole
    (1, 3, 281, 279, 17, 3, 1, 1, 1),    # 32 x 128, staged through registers
    (2, 4, 200, 201, 33, 3, 1, 1, 1),    # one slice
    (1, 36, 104, 104, 65, 3, 1, 1, 1),   # 64 x 128, split k range of several slices with a short last one
    (3, 64, 19, 19, 70, 3, 1, 1, 1),     # 64 x 64, split k range, pixels of two images in one group of four
    (1, 1024, 4, 4, 255, 1, 1, 0, 1),    # split, planes of 16
    (2, 20, 13, 11, 65, 3, 2, 1, 1),
    (1, 7, 20, 23, 9, 5, 2, 2, 1),       # any kernel size
    (1, 3, 21, 25, 4, 3, 1, 2, 2),       # dilated
    (1, 9, 21, 25, 12, 3, 1, 2, 2),      # dilated, beyond the little work that the per-tap kernel takes
    (2, 3, 90, 100, 4, 5, 1, 2, 1),      # four filters of a general kernel, an image too small for the per-tap kernel
    (1, 2, 200, 190, 3, 5, 1, 2, 1),     # three, large enough
    (1, 16, 256, 257, 1, 3, 1, 1, 1),    # one 3x3 filter on a large image
    (1, 1, 300, 220, 1, 1, 1, 0, 1),     # one product
    (1, 4, 32, 32, 62, 3, 1, 1, 1),      # 36 products, a last group of two filters
    (1, 2, 24, 24, 3, 9, 1, 4, 1),       # more than 64 taps
    (1, 1, 1, 1, 1, 1, 1, 0, 1),
])
def test_conv2d_f32_tiles(be, geom):
    B, C, H, W, F, k, s, pad, dil = geom
    rng = np.random.default_rng(C + F)
    x = rng.normal(0, 1, (B, C, H, W)).astype(np.float32)
    w = rng.normal(0, 1, (F, C, k, k)).astype(np.float32)
    oh, ow = (H + 2 * pad - k) // s + 1, (W + 2 * pad - k) // s + 1  # (dilation does not enter the extent)
    t = be.conv2d_f32(be.upload_f32(x.shape, x), be.upload_f32(w.shape, w), (B, F, oh, ow), C, H, W, F, k, s, s, dil, pad, 1)
    got = be.download_f32(t).astype(np.float64)
    grow = dil * (k - 1) + 1 - k  # the reference's extent ignores dilation: extend the input so that every tap exists as a zero
    xd = torch.nn.functional.pad(torch.from_numpy(x).double(), (pad, pad + grow, pad, pad + grow))
    wd = torch.from_numpy(w).double()
    ref = torch.nn.functional.conv2d(xd, wd, stride=s, dilation=dil)[:, :, :oh, :ow].numpy()
    size = torch.nn.functional.conv2d(xd.abs(), wd.abs(), stride=s, dilation=dil)[:, :, :oh, :ow].numpy()
    # one rounding of 2^-24 per term of the chain, at most C k^2 of them and the sums over the parts of a split range
    assert (np.abs(got - ref) <= (C * k * k + 33) * 2.0 ** -24 * size).all()


@pytest.mark.parametrize("filters", [64 * 65535, 64 * 65535 + 1])
def test_conv2d_f32_millions_of_filters(be, filters):
    """The last filter tile that the grid of the blocked kernel numbers, and one filter more: a product per output, the same bits."""
    w = np.random.default_rng(1).normal(0, 1, filters).astype(np.float32)
    t = be.conv2d_f32(be.upload_f32((1, 1, 1, 1), np.full(1, 1.5, np.float32)), be.upload_f32((filters, 1, 1, 1), w), (1, filters, 1, 1), 1, 1, 1, filters, 1, 1, 1, 1, 0, 1)
    np.testing.assert_array_equal(be.download_f32(t).ravel(), w * np.float32(1.5))


@pytest.mark.parametrize("filters", [3, 40])
def test_conv2d_f32_dilation_far_beyond_the_image(be, filters):
    """Only tap (0, 0) lies inside; the pixels of the tile behind the last output read nothing, however far the dilation reaches."""
    rng = np.random.default_rng(filters)
    x, w = rng.normal(0, 1, (1, 5, 5, 6)).astype(np.float32), rng.normal(0, 1, (filters, 5, 3, 3)).astype(np.float32)
    t = be.conv2d_f32(be.upload_f32(x.shape, x), be.upload_f32(w.shape, w), (1, filters, 3, 4), 5, 5, 6, filters, 3, 1, 1, 1 << 27, 0, 1)
    ref = np.einsum("fc,chw->fhw", w[:, :, 0, 0].astype(np.float64), x[0, :, :3, :4].astype(np.float64))
    assert (np.abs(be.download_f32(t)[0] - ref) <= 78 * 2.0 ** -24 * 5 * np.abs(x).max() * np.abs(w).max()).all()


def test_calibrated_scales_do_not_depend_on_the_batch(be):
    """One image, alone and eight times in a batch: the f32 convolutions cut their work differently, the scales stay bit for bit."""
    import lightnet_b200 as ln
    from lightnet_b200 import synth, zoo
    x = synth.uniform_images(1, 3, 96, 160, 5)
    scales = []
    for batch in (1, 8):
        net = ln.GpuExecutableNetwork(be, zoo.yolov3_tiny_cfg(160, 96), batch, ln.LN_Q8)
        net.load_weights(synth.he_weights(net.layers(), 3))
        net.calibrate(np.repeat(x, batch, 0))
        scales.append(np.asarray(net.scales()))
    np.testing.assert_array_equal(scales[0], scales[1])


@pytest.mark.parametrize("geom", [
    (1, 36, 26, 26, 65, 3, 1, 1, 1),     # blocked, split k range
    (2, 32, 160, 160, 128, 3, 1, 1, 1),  # 64 x 128 tiles
    (1, 5, 30, 31, 17, 3, 2, 1, 1),      # staged through registers
    (1, 3, 30, 31, 17, 3, 2, 1, 1),      # per tap
    (1, 5, 13, 13, 40, 3, 1, 1, 1),      # k range not a multiple of 4
    (2, 64, 9, 9, 70, 1, 1, 1, 1),       # 1x1 with padding: border outputs have no tap at all
    (1, 7, 12, 14, 9, 5, 1, 2, 1),
    (1, 6, 15, 17, 4, 3, 1, 2, 2),       # dilated
    (1, 4, 11, 10, 8, 3, 1, 1, 1, 2),    # grouped
])
def test_conv2d_f32_weights_that_are_not_finite(be, geom):
    """Taps outside the image are skipped, so an infinite or NaN weight on them leaves the output alone: the same outputs are NaN, +inf and -inf as
    in a sum over the taps inside, and the finite ones agree."""
    B, C, H, W, F, k, s, pad, dil = geom[:9]
    groups = geom[9] if len(geom) > 9 else 1
    rng = np.random.default_rng(C + F)
    x = rng.normal(0, 1, (B, C, H, W)).astype(np.float32)
    w = rng.normal(0, 1, (F, C // groups, k, k)).astype(np.float32)
    for f, tap, v in ((0, 0, np.inf), (1, 0, -np.inf), (2, k * k - 1, np.nan), (3, k * k // 2, np.inf), (F - 1, k * k - 1, np.inf)):
        w[f, f % (C // groups), tap // k, tap % k] = v
    oh, ow = (H + 2 * pad - k) // s + 1, (W + 2 * pad - k) // s + 1
    got = be.download_f32(be.conv2d_f32(be.upload_f32(x.shape, x), be.upload_f32(w.shape, w), (B, F, oh, ow), C, H, W, F, k, s, s, dil, pad, groups)).astype(np.float64)
    ref, size = np.zeros((B, F, oh, ow)), np.zeros((B, F, oh, ow))
    fpg, cpg = F // groups, C // groups
    with np.errstate(invalid="ignore"):
        for ky in range(k):
            for kx in range(k):
                ys, xs = np.arange(oh) * s + ky * dil - pad, np.arange(ow) * s + kx * dil - pad
                iy, ix = np.flatnonzero((ys >= 0) & (ys < H)), np.flatnonzero((xs >= 0) & (xs < W))
                if not len(iy) or not len(ix):
                    continue
                patch = x[:, :, ys[iy]][:, :, :, xs[ix]].astype(np.float64)
                for f in range(F):
                    term = w[f, :, ky, kx].astype(np.float64)[None, :, None, None] * patch[:, f // fpg * cpg:(f // fpg + 1) * cpg]
                    ref[:, f, iy[0]:iy[-1] + 1, ix[0]:ix[-1] + 1] += term.sum(1)
                    size[:, f, iy[0]:iy[-1] + 1, ix[0]:ix[-1] + 1] += np.abs(term).sum(1)
    np.testing.assert_array_equal(np.isnan(got), np.isnan(ref))
    np.testing.assert_array_equal(np.isinf(got) * np.sign(np.nan_to_num(got)), np.isinf(ref) * np.sign(np.nan_to_num(ref)))
    ok = np.isfinite(ref)
    assert (np.abs(got[ok] - ref[ok]) <= (C * k * k + 33) * 2.0 ** -24 * size[ok]).all()


@pytest.mark.parametrize("geom", [(512, 13, 13, 256, 3), (256, 26, 20, 512, 1), (1024, 4, 4, 255, 1), (68, 19, 21, 40, 3), (7, 20, 23, 9, 5), (35, 30, 30, 17, 3),
                                  (2, 60, 60, 16, 3), (1, 40, 41, 2, 5), (3, 90, 95, 1, 5), (3, 60, 65, 4, 7), (1, 120, 100, 1, 3)])  # where the choice of the kernel looks at sizes
def test_conv2d_f32_does_not_depend_on_the_batch(be, geom):
    """An image has the same bits alone and as any of 2, 9 or 40 images: the order of a sum is cut by the size of one image."""
    C, H, W, F, k = geom
    rng = np.random.default_rng(C)
    x, w = rng.normal(0, 1, (2, C, H, W)).astype(np.float32), rng.normal(0, 1, (F, C, k, k)).astype(np.float32)
    tw = be.upload_f32(w.shape, w)

    def conv(x):
        x = np.ascontiguousarray(x)
        return be.download_f32(be.conv2d_f32(be.upload_f32(x.shape, x), tw, (len(x), F, H, W), C, H, W, F, k, 1, 1, 1, k // 2, 1))

    alone = np.concatenate([conv(x[:1]), conv(x[1:])])
    for n in (2, 9, 40):
        got = conv(np.resize(x, (n, C, H, W)))
        np.testing.assert_array_equal(got, np.resize(alone, got.shape))


def test_f32_heads_do_not_depend_on_the_batch(be):
    import lightnet_b200 as ln
    from lightnet_b200 import synth, zoo
    x = synth.uniform_images(1, 3, 160, 224, 5)
    heads = []
    for batch in (1, 12):
        net = ln.GpuExecutableNetwork(be, zoo.yolov3_tiny_cfg(224, 160), batch, ln.LN_F32)
        net.load_weights(synth.he_weights(net.layers(), 3))
        net.forward(np.repeat(x, batch, 0))
        heads.append([be.download_f32(net.head(k)) for k in range(net.num_heads())])
    for a, b in zip(*heads):
        np.testing.assert_array_equal(np.repeat(a, 12, 0), b)
