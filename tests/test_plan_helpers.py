"""Host-side planner helpers of the convolution kernel, compiled with g++ from the header they live in (no GPU)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INCLUDE = "/usr/local/cuda/include"

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "ln_conv_plan.h"
int main(int argc, char** argv) {
    for (int i = 1; i + 3 < argc; i += 4)
        printf("%d\n", ln_acc_shift((float)atof(argv[i]), (float)atof(argv[i + 1]), (float)atof(argv[i + 2]), (float)atof(argv[i + 3])));
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None or not os.path.isdir(CUDA_INCLUDE), reason="needs g++ and the CUDA headers")
def test_acc_shift_rule(tmp_path):
    """ln_acc_shift: 0 while 127 * max_l1 stays below 2^22; otherwise the smallest shift that brings the bound under 2^22, allowed
    only while half of what is dropped (2^(shift-1) accumulator units) times the largest multiplier s_x * s_w / s_y stays at or
    under 0.02 of a code; -1 when that fails or more than 8 bits would be needed."""
    src = tmp_path / "acc_shift.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "acc_shift"
    subprocess.run(["g++", "-std=c++17", "-I" + CUDA_INCLUDE, "-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(ROOT, "lightnet_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    cases = [
        # max_l1, s_x, max s_w, 1 / s_y  ->  expected
        ((1000.0, 0.01, 0.001, 10.0), 0),          # 127 k < 2^22
        ((33025.0, 0.01, 0.001, 10.0), 0),         # 4 194 175 < 2^22: still none
        ((33027.0, 0.01, 0.001, 10.0), 1),         # just above: one bit, costs 1 * 1e-4 codes
        ((33027.0, 1.0, 0.5, 1.0), -1),            # one bit would cost half a code
        ((143000.0, 0.02, 0.002, 8.0), 3),         # 18.2 M < 2^25: three bits, 4 * 3.2e-4 codes
        ((143000.0, 0.02, 0.002, 20.0), 3),        # 4 * 8e-4 = 0.0032
        ((143000.0, 0.2, 0.01, 10.0), -1),         # 4 * 0.02 = 0.08 of a code: refused
        ((8.0e6, 1e-4, 1e-4, 1.0), 8),             # 1.016e9 < 2^30
        ((2.0e7, 1e-4, 1e-4, 1.0), -1),            # beyond 2^30: nothing up to eight bits is enough
    ]
    args = [repr(float(v)) for c, _ in cases for v in c]
    out = subprocess.run([str(exe)] + args, check=True, capture_output=True, text=True).stdout.split()
    assert [int(v) for v in out] == [want for _, want in cases]


F32_PROGRAM = r"""
#include <cstdio>
#include "ln_conv_f32_plan.h"
int main() {
    // n, c, h, w, f, k, oh, ow
    printf("%d", ln_conv_f32_blocked(1, 1, 46400, 46400, 1, 1, 23200, 23200));  // a plane beyond 2^31 values, read with a stride
    printf("%d", ln_conv_f32_blocked(1, 1, 46340, 46340, 1, 1, 23170, 23170));  // just below
    printf("%d", ln_conv_f32_blocked(1, 3, 46400, 46400, 8, 3, 11600, 11600));
    printf("%d", ln_conv_f32_blocked(1, 1, 32768, 32768, 1, 1, 32768, 32768));  // 2^30 output pixels
    printf("%d", ln_conv_f32_blocked(4, 1 << 22, 1, 1, 8, 2, 1, 1));            // k range of 2^24
    printf("%d", ln_conv_f32_blocked(1, 1, 1, 1, 64 * 65535, 1, 1, 1));         // the last filter tile of the grid, and one more
    printf("%d", ln_conv_f32_blocked(1, 1, 1, 1, 64 * 65535 + 1, 1, 1, 1));
    printf("%d\n", ln_conv_f32_blocked(64, 512, 19, 19, 1024, 3, 19, 19));
    return 0;
}
"""


def _run(tmp_path, program):
    src, exe = tmp_path / "p.cpp", tmp_path / "p"
    src.write_text(program)
    subprocess.run(["g++", "-std=c++17", "-I" + os.path.join(ROOT, "lightnet_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    return subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_f32_convolutions_beyond_32_bit_indices_are_not_blocked(tmp_path):
    assert _run(tmp_path, F32_PROGRAM) == ["01000101"]


F32_CUT_PROGRAM = r"""
#include <cstdio>
#include <initializer_list>
#include "ln_conv_f32_plan.h"
int main() {
    long split = 0, uneven = 0;
    for (int ks : {0, 1, 3})
        for (int async = 0; async <= (ks ? 1 : 0); ++async)
            for (long F : {8, 33, 70, 255, 512})
                for (long plane : {1, 49, 361, 1444, 23104})
                    for (long images : {1, 3, 16})
                        for (int c = 4; c <= 1100; c += c < 80 ? 4 : 52) {
                            const int K = c * (ks == 1 ? 1 : 9), SL = ln_conv_f32_slice(async, ks), slices = (K + SL - 1) / SL;
                            if (async && F <= 32) continue;
                            const ln_conv_f32_cut cut = ln_conv_f32_choose(148, images, plane, F, K, ks, async, false);
                            split += cut.parts > 1;
                            int most = 0, least = 1 << 30;
                            for (int z = 0; z < cut.parts; ++z) {
                                const int n = ln_conv_f32_first_slice(slices, z + 1, cut.parts) - ln_conv_f32_first_slice(slices, z, cut.parts);
                                most = n > most ? n : most;
                                least = n < least ? n : least;
                            }
                            uneven += most != least;
                            if (ln_conv_f32_first_slice(slices, 0, cut.parts) != 0 || ln_conv_f32_first_slice(slices, cut.parts, cut.parts) != slices || least < 1 || most - least > 1 ||
                                (cut.parts > 1 && (K < 64 || least < (async ? 2 : 4))) || ln_conv_f32_choose(148, images, plane, F, K, ks, async, true).parts != 1) {
                                printf("ks %d async %d F %ld plane %ld images %ld c %d: %d parts of %d to %d slices\n", ks, async, F, plane, images, c, cut.parts, least, most);
                                return 0;
                            }
                        }
    printf("%d\n", split > 500 && uneven > 200);
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_f32_k_ranges_are_split_evenly(tmp_path):
    """Every CTA of a cluster has slices to sum, as many as the others or one more or less; sums of less than 64 products stay whole."""
    assert _run(tmp_path, F32_CUT_PROGRAM) == ["1"]
