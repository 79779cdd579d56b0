"""The small-grid form of the tensor-core convolution (short chains, k range split over clusters) against the persistent form and a
float64 convolution, at the edges of its tiles, stages and splits."""
import os
import shutil
import subprocess

import numpy as np
import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INCLUDE = "/usr/local/cuda/include"

# batch, channels, height, width, filters, kernel, stride, padding
CASES = [
    (1, 512, 8, 16, 64, 3, 1, 1),     # one tile, 36 k-blocks over eight CTAs (five and four each)
    (1, 1100, 5, 7, 32, 3, 1, 1),     # channels padded, one 32-filter tile over four CTAs
    (1, 256, 13, 13, 255, 1, 1, 0),   # ragged filters: a last chunk with one filter missing
    (2, 160, 19, 19, 96, 3, 2, 1),    # 32-byte channel blocks, three filter tiles of 32, stride 2
    (1, 64, 9, 11, 40, 3, 1, 1),      # 64-byte channel blocks, zero-padded second filter tile
    (3, 32, 20, 24, 64, 1, 1, 0),     # pixel groups
    (1, 1024, 19, 19, 512, 1, 1, 0),  # split, several pixel tiles
    (1, 32, 1, 1, 32, 1, 1, 0),       # one k-block, one pixel
    (4, 256, 61, 61, 128, 3, 1, 1),   # 128-filter tiles: a ring of three stages shared by two issuers, 18 k-blocks
    (1, 512, 38, 38, 256, 3, 1, 1),   # the same over 36
]


@pytest.fixture(scope="module")
def be():
    import lightnet_b200 as ln
    b = ln.B200Backend(0)
    yield b
    b.close()


def _both(monkeypatch, call):
    got = []
    for off in ("", "small"):
        monkeypatch.setenv("LN_CONV_DISABLE", off)
        got.append(call())
    return got


def _reference(x, w, s, p):
    return torch.nn.functional.conv2d(torch.from_numpy(x).double(), torch.from_numpy(w).double(), stride=s, padding=p).numpy()


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["int8", "fp8"])
@pytest.mark.parametrize("case", CASES)
def test_small_grid_8_bit(be, monkeypatch, case, kind):
    import lightnet_b200 as ln
    n, c, h, w, f, k, s, p = case
    dtype = ln.LN_Q8 if kind == "int8" else ln.LN_F8
    rng = np.random.default_rng(c + f)
    x, wt = rng.normal(0, 1, (n, c, h, w)).astype(np.float32), rng.normal(0, 1, (f, c, k, k)).astype(np.float32)
    shape = (n, f, (h + 2 * p - k) // s + 1, (w + 2 * p - k) // s + 1)
    wq, tx = be.conv_weights_q(be.upload_f32(wt.shape, wt), f, c, k, dtype), be.upload_q(x.shape, x, 4.0 / (127.0 if kind == "int8" else 448.0), dtype)
    bias = be.upload_f32((1, f, 1, 1), rng.normal(0, 1, f).astype(np.float32))

    def conv(act, scale, out):
        return be.conv2d_bias_act_q(tx, wq, bias, shape, c, h, w, f, k, s, s, 1, p, 1, act, scale, out)

    if kind == "int8":
        codes = np.clip(np.rint(wt / (np.abs(wt.reshape(f, -1)).max(1) / np.float32(127.0))[:, None, None, None]), -127, 127)
        ref = _reference(be.download_q(tx)[0].astype(np.float32), codes.astype(np.float32), s, p)
        for acc in _both(monkeypatch, lambda: be.download_i32(conv("linear", 1.0, ln.LN_OUT_ACC))):
            np.testing.assert_array_equal(acc, ref)
    # the same accumulators through the same epilogue: the same codes and the same head values
    for act in ("leaky", "mish"):
        a, b = _both(monkeypatch, lambda: be.download_q(conv(act, 0.5, ln.LN_OUT_Q))[0])
        np.testing.assert_array_equal(a, b)
    a, b = _both(monkeypatch, lambda: be.download_f32(conv("linear", 1.0, ln.LN_OUT_F32)))
    np.testing.assert_array_equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES)
def test_small_grid_f16(be, monkeypatch, case):
    n, c, h, w, f, k, s, p = case
    rng = np.random.default_rng(c + f)
    x = rng.normal(0, 1, (n, c, h, w)).astype(np.float16).astype(np.float32)
    wt = (rng.normal(0, 1, (f, c, k, k)) / np.sqrt(c * k * k)).astype(np.float16).astype(np.float32)
    shape = (n, f, (h + 2 * p - k) // s + 1, (w + 2 * p - k) // s + 1)
    ref, size = _reference(x, wt, s, p), _reference(np.abs(x), np.abs(wt), s, p)
    bias = be.upload_f32((1, f, 1, 1), np.zeros(f, np.float32))
    tx = be.upload_f16(x.shape, x)

    def conv():
        wh = be.conv_weights_f16(be.upload_f32(wt.shape, wt), f, c * k * k)
        return be.download_f16(be.conv2d_bias_act_f16(tx, wh, bias, shape, c, h, w, f, k, s, s, 1, p, 1, "linear"))

    # one rounding to 11 bits of the result, binary32 accumulation: 2^-13 of the sum of magnitudes (the bound of the 8-bit float tests)
    pair = _both(monkeypatch, conv)
    np.testing.assert_array_equal(pair[0], pair[1])  # one chain per output in either form
    for got in pair:
        assert (np.abs(got - ref) <= 2.0 ** -11 * np.abs(ref) + 2.0 ** -13 * size + 2.0 ** -24).all()


@pytest.mark.gpu
@pytest.mark.parametrize("model,kind", [("yolov4", "int8"), ("yolov4", "fp8"), ("yolov7", "fp8")])
@pytest.mark.parametrize("exact", [False, True])
def test_small_grid_networks_layer_by_layer(be, monkeypatch, capfd, model, kind, exact):
    """Plans of a network, layer by layer against the persistent kernel's: space-to-depth input, pixel groups of 1x1 and 3x3 layers, fused shortcuts
    (int8), inputs and outputs that are channel slices of a concatenated buffer."""
    import lightnet_b200 as ln
    from lightnet_b200 import synth, zoo
    cfg = (zoo.yolov4_cfg if model == "yolov4" else zoo.yolov7_cfg)(192, 160).replace("activation=logistic", "activation=linear")
    prec = ln.LN_Q8 if kind == "int8" else ln.LN_F8
    x = synth.uniform_images(2, 3, 160, 192, 9)
    outs, plans, scales = [], [], None
    monkeypatch.setenv("LN_DEBUG_PLAN", "1")
    be.set_exact_epilogue(exact)
    try:
        for off in ("", "small"):
            monkeypatch.setenv("LN_CONV_DISABLE", off)
            net = ln.GpuExecutableNetwork(be, cfg, 2, prec)
            net.load_weights(synth.he_weights(net.layers(), 3))
            if scales is None:
                net.calibrate(x)
                scales = net.scales()
            net.set_scales(scales)
            capfd.readouterr()
            net.forward(x)
            plans.append([line for line in capfd.readouterr().err.splitlines() if line.startswith("plan:")])
            got, fused = {}, 0
            for i, layer in enumerate(net.layers()):
                try:
                    t = net.layer_output(i)
                except ln.BackendError as e:
                    assert e.kind == "unsupported"  # fused into the layer after it, or kept in space-to-depth layout
                    fused += 1
                    continue
                got[i] = be.download_f32(t) if t.dtype == ln.LN_F32 else be.download_q(t)[0]
            outs.append(got)
            del net
    finally:
        be.set_exact_epilogue(False)
    small = [line for line in plans[0] if "small grid" in line]
    assert len(small) > 40 and not any("small grid" in line for line in plans[1])
    assert any("pack 4" in line or "pack 2" in line for line in small)
    assert model != "yolov4" or any("bk 64" in line and "pack 2" in line for line in small)  # two pixels of 32 channels per row: a 3x3 layer
    assert fused >= (20 if model == "yolov4" and kind == "int8" else 1 if model == "yolov4" else 0)
    assert outs[0].keys() == outs[1].keys()
    for i in outs[0]:
        np.testing.assert_array_equal(outs[0][i], outs[1][i], err_msg="layer %d" % i)


PROGRAM = r"""
#include <cstdio>
#include "ln_conv_plan.h"
int main() {
    long n = 0, split = 0, padded = 0;
    for (int kind = 0; kind < 3; ++kind)
        for (int m = 1; m <= 400; m += m < 8 ? 1 : 7)
            for (int F = 1; F <= 1100; F += F < 300 ? 31 : 97)
                for (int bk = 32; bk <= 128; bk *= 2)
                    for (int kb = 1; kb <= 72; kb += kb < 9 ? 1 : 9) {
                        const int fpad = (int)ln_round_up(F, ln_conv_choose_bn(F));
                        int bn = 0, ks = 0;
                        if (!ln_conv_choose_small(148, kind, m, F, fpad, kb, bk, &bn, &ks)) {
                            const int wide = fpad % 128 == 0 ? 128 : (fpad % 64 == 0 ? 64 : 32);
                            if ((long)m * ((F + wide - 1) / wide) <= 296) { printf("refused m %d F %d\n", m, F); return 1; }
                            continue;
                        }
                        ++n;
                        split += ks > 1;
                        const long tiles = (long)m * ((F + bn - 1) / bn);
                        if (fpad % bn || bn > 128 || bn < 32 || (ks & (ks - 1)) || ks < 1 || ks > 8 || tiles * ks > 296 || ks > kb || bn / 8 % ks || (kind != LN_KIND_I8 && ks > 1)) {
                            printf("bad choice kind %d m %d F %d kb %d bk %d: bn %d ks %d\n", kind, m, F, kb, bk, bn, ks);
                            return 1;
                        }
                        // two CTAs fit an SM (228 KB, 1 KB of it per CTA), and three of a cluster launch never do: each may hold half of its TMEM
                        int stages = 0, region = 0;
                        const long smem = (long)ln_conv_small_smem(bk, bn, ks, kb, &stages, &region), sm = 228 * 1024;
                        padded += smem > region + 1024 + (long)kSmallBarBytes + bn * 8;
                        if (2 * (smem + 1024) > sm || (ks > 1 && 3 * (smem + 1024) <= sm) || stages < 1 || stages > kMaxStages || region < stages * (128 + bn) * bk ||
                            (ks > 1 && region < bn / 8 * (long)kPieceBytes) || smem < region + 1024 + (long)kSmallBarBytes + bn * 8) {
                            printf("bad shared memory: bn %d ks %d kb %d bk %d: %ld bytes, %d stages, region %d\n", bn, ks, kb, bk, smem, stages, region);
                            return 1;
                        }
                    }
    printf("%d\n", n > 1000 && split > 100 && padded > 0);
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None or not os.path.isdir(CUDA_INCLUDE), reason="needs g++ and the CUDA headers")
def test_choice_of_tile_and_split(tmp_path):
    """Every choice of the planner is one the kernel can run: whole filter tiles, at least one k-block and one piece per CTA, two CTAs per SM."""
    src, exe = tmp_path / "small.cpp", tmp_path / "small"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I" + CUDA_INCLUDE, "-I" + os.path.join(ROOT, "include"), "-I" + os.path.join(ROOT, "lightnet_b200", "csrc"), str(src),
                    "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip() == "1", out.stdout
