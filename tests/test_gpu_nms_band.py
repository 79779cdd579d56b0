"""Decode + NMS at the edges of its sort, chunks and class buckets: the records must be the oracle's, whichever way the candidates
reach the band (all at once at an ordinary threshold, through the histogram of the heads below it)."""
import numpy as np
import pytest

from oracle import oracle_api as orc

pytestmark = pytest.mark.gpu
ANCH = [(10.0, 13.0), (16.0, 30.0), (33.0, 23.0)]


@pytest.fixture(scope="module")
def be():
    import lightnet_b200 as ln
    b = ln.B200Backend(0)
    yield b
    b.close()


# candidates of the image: none, one, around a warp, a chunk of 512, each size class of the sort, and more than a band holds (16384)
@pytest.mark.parametrize("n", [0, 1, 31, 33, 511, 512, 513, 1025, 2049, 4097, 8193, 16385])
@pytest.mark.parametrize("classes", [1, 300])  # one bucket for everything / several classes per bucket
@pytest.mark.parametrize("thr", [0.1, 0.01])
def test_band_edges(be, n, classes, thr):
    g = 76
    rng = np.random.default_rng(n + classes)
    v = np.full((1, 3, 5 + classes, g * g), -12.0, np.float32)
    v[:, :, 0:2] = rng.normal(0, 2, (1, 3, 2, g * g))
    v[:, :, 2:4] = rng.normal(0.5, 0.7, (1, 3, 2, g * g))
    slots = rng.permutation(3 * g * g)[:n]
    a, cell = slots // (g * g), slots % (g * g)
    v[0, a, 4, cell] = 3.0
    v[0, a, 5 + rng.integers(0, classes, n), cell] = np.round(rng.normal(1.0, 0.7, n), 1)  # rounded: plenty of equal scores
    h = v.reshape(1, 3 * (5 + classes), g, g)
    specs = [dict(gw=g, gh=g, classes=classes, anchors=ANCH, scale_x_y=1.0, new_coords=0)]
    dev = [dict(raw=be.upload_f32(h.shape, h), classes=classes, anchors=ANCH, scale_x_y=1.0, new_coords=0)]
    recs = orc.decode_only([h[0]], specs, 608, 608, 640, 480, thr, letterbox=True, det_exp=True)
    assert recs.shape[0] == n
    for max_per_image in (300, 4096):
        got = be.yolo_decode_nms(dev, 608, 608, 640, 480, thr, 0.45, True, 0, max_per_image)[0]
        ref = orc.nms_records_first_k(recs, 0.45, max_per_image)
        assert got.shape == ref.shape and np.array_equal(got, ref)
