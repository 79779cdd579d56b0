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
