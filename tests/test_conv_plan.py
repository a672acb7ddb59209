"""How the network's convolutions are cut (nn/conv_plan.h), compiled here and
asked for shapes."""
import os
import subprocess

import pytest

from mplb_b200 import build

SOURCE = r"""
#include <cstdio>
#include <cstring>
#include "conv_plan.h"
using namespace mplb::nn;
int main() {
    char what[16];
    int n, h, w, cin, cout;
    while (scanf("%15s %d %d %d %d %d", what, &n, &h, &w, &cin, &cout) == 6)
        if (!strcmp(what, "band"))
            printf("%d\n", PlanBand(n, h, w, cin, cout, 148).tiles);
        else {
            const WgradBandPlan p = PlanWgradBand(n, h, w, cin, cout, 148);
            printf("%d %d %d %d %d %d %d %d %d %d\n", p.bn, p.slices, p.groups,
                   p.rows, p.bands_per_img, p.bands_per_cta, p.ctas, p.stages,
                   WgradBandSmem(w, p.rows, p.stages, p.bn),
                   128 * WgradTapBlocks((long long)n * h * w / 128, 9, cin,
                                        cout, 148));
        }
}
"""


@pytest.fixture(scope="module")
def ask(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "ask.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I",
                    os.path.join(build.CSRC, "nn"), "-o", d / "ask",
                    d / "ask.cpp"], check=True)

    def run(what, shapes):
        text = "".join(f"{what} {' '.join(map(str, s))}\n" for s in shapes)
        out = subprocess.run([d / "ask"], input=text, capture_output=True,
                             text=True, check=True).stdout
        return [list(map(int, line.split())) for line in out.splitlines()]
    return run


# images, height, width, input and output channels; microseconds of the launch
# tap by tap and in bands (B200, cold caches)
TIMES = [
    (512, 128, 1, 96, 64, 18.7, 31.8), (64, 128, 1, 128, 384, 14.5, 28.4),
    (128, 128, 1, 64, 128, 9.0, 16.0), (4096, 128, 1, 16, 16, 73.5, 53.8),
    (4096, 64, 2, 128, 192, 330.0, 426.3), (512, 64, 2, 96, 192, 38.6, 54.2),
    (16, 32, 4, 128, 96, 11.5, 8.7), (4096, 32, 4, 32, 128, 100.2, 150.5),
    (512, 16, 8, 128, 384, 84.7, 127.9), (512, 16, 8, 96, 32, 17.2, 23.4),
    (32, 16, 16, 128, 256, 13.5, 17.6), (64, 16, 16, 128, 256, 13.9, 28.3),
    (8, 16, 16, 80, 160, 15.5, 11.2), (2, 32, 32, 32, 128, 8.0, 6.2),
    (32, 32, 32, 128, 96, 21.6, 16.7), (8, 32, 32, 128, 384, 14.4, 19.3),
    (512, 32, 32, 16, 32, 71.7, 32.1), (2, 64, 64, 48, 48, 11.0, 8.3),
    (16, 64, 64, 128, 256, 48.2, 77.5), (8, 64, 64, 96, 32, 15.5, 12.2),
    (2, 128, 128, 128, 96, 21.7, 15.5), (8, 128, 128, 16, 32, 22.1, 13.7),
    (32, 128, 128, 32, 32, 45.6, 28.4),
]


def test_the_faster_form_is_taken(ask):
    """Shapes whose two forms are more than a quarter apart."""
    for row, (tiles,) in zip(TIMES, ask("band", [r[:5] for r in TIMES])):
        assert max(row[5:]) > 1.25 * min(row[5:])
        assert (tiles > 0) == (row[6] < row[5]), row


def test_wide_inputs_go_tap_by_tap(ask):
    assert ask("band", [(32, 64, 64, 144, 64), (1, 16, 16, 384, 16)]) == [[0]] * 2


WGRAD = [(n, h, w, ci, co)
         for n in (1, 2, 3, 5, 8, 20, 32, 64, 100)
         for h, w in ((16, 16), (24, 16), (32, 32), (36, 32), (64, 64), (6, 64),
                      (128, 128), (1, 128), (9, 128), (1000, 32))
         for ci, co in ((32, 32), (96, 32), (16, 48), (32, 64), (64, 64),
                        (192, 64), (64, 128), (128, 128), (384, 128),
                        (128, 256), (256, 256), (5000, 16))]


def test_weight_gradient_bands(ask):
    """Bands cover every image in even heights, fit in shared memory, and no
    accumulator sums more pixels than those of the tap-by-tap kernels (their
    fp32 error grows with the number), or than twice an SM's share of a group
    of output channels."""
    for shape, got in zip(WGRAD, ask("wgrad", WGRAD)):
        n, h, w, ci, co = shape
        bn, slices, groups, rows, per_img, per_cta, ctas, stages, smem, tap = got
        assert bn * groups >= co and 32 * slices >= ci
        assert rows >= 1 and per_img == -(-h // rows), shape
        assert rows == -(-h // per_img) and rows <= 250
        assert ctas == -(-n * per_img // per_cta)
        assert 2 <= stages <= 4 and smem <= 227 * 1024
        assert rows * per_cta * w <= tap, shape
        share = 2 * n * h * w * slices // 148
        assert rows * per_cta * w <= max(128, share), shape
        # enough pixels to pay for the sums' way out, where there are any
        assert rows * per_cta * w >= min(128, n * h * w), shape


def test_weight_gradients_fill_the_gpu(ask):
    """The network's layers at 32 and 8 images: CTAs for nine tenths of the
    SMs, or of the last round of them."""
    layers = [(128, 32, 32), (128, 96, 32), (64, 32, 64), (64, 64, 64),
              (64, 192, 64), (32, 128, 128), (32, 384, 128)]
    shapes = [(n, s, s, ci, co) for n in (8, 32) for s, ci, co in layers]
    for shape, got in zip(shapes, ask("wgrad", shapes)):
        ctas = got[6] * got[1] * got[2]
        rounds = -(-ctas // 148)
        assert ctas >= 0.85 * 148 * rounds, (shape, ctas)
