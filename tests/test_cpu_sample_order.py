"""The order in which an image's samples are generated, compiled for the host:
every sample of every pixel once, and no long stretch of few pixels (samples that
finish together add to the film one after the other where they share a pixel)."""
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
struct float4;
#include "ar_types.h"
#include <cstdio>
#include <cstdlib>
int main(int argc, char** argv) {
    const unsigned npix = strtoul(argv[1], 0, 10), spp = strtoul(argv[2], 0, 10);
    const unsigned long long total = (unsigned long long)npix * spp, from = strtoull(argv[3], 0, 10);
    const unsigned long long n = strtoull(argv[4], 0, 10);
    for (unsigned long long g = from; g < from + n && g < total; ++g) {
        const ar::PixelSample p = ar::pixel_sample(g, npix, spp);
        const unsigned w[2] = {p.pixel, p.sample};
        fwrite(w, 4, 2, stdout);
    }
}
"""


@pytest.fixture(scope="module")
def order(tmp_path_factory):
    d = tmp_path_factory.mktemp("order")
    src, exe = d / "order.cpp", d / "order"
    src.write_text(PROGRAM)
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "agent-ray_b200", "csrc"), "-o", str(exe), str(src)])

    def run(npix, spp, first=0, count=1 << 62):
        out = subprocess.check_output([str(exe), str(npix), str(spp), str(first), str(count)])
        return np.frombuffer(out, np.uint32).reshape(-1, 2)
    return run


@pytest.mark.parametrize("npix", [1, 7, 1024, 1025, 3001])
@pytest.mark.parametrize("spp", [1, 3, 4, 5, 63, 64, 65, 130])
def test_every_sample_once_and_pixels_spread(order, npix, spp):
    ps = order(npix, spp).astype(np.int64)
    assert len(ps) == npix * spp and ps[:, 0].max() < npix and ps[:, 1].max() < spp
    assert len(np.unique(ps[:, 0] * spp + ps[:, 1])) == npix * spp
    window = 64 * 100
    for first in range(0, len(ps) - window, window // 2):
        assert len(np.unique(ps[first:first + window, 0])) >= min(npix, 100)


def test_large_images_and_sample_counts(order):
    # 64-bit numbers: the last samples of 60000 x 60000 pixels and of 2^31 samples
    for npix, spp in ((3_600_000_000, 100), (2000, 1 << 31), (1, (1 << 32) - 1)):
        ps = order(npix, spp, npix * spp - 4, 4)
        assert ps[-1].tolist() == [npix - 1, spp - 1]
        assert len(np.unique(ps, axis=0)) == 4
