"""Layout of the scene's geometry buffer, compiled for the host: sections that
do not overlap, and links that reach what a GPU's memory holds."""
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
struct float4;
#include "bvh_build.hpp"
#include <cstdio>
#include <cstdlib>
using namespace ar;
int main(int argc, char** argv) {
    for (int k = 1; k + 2 < argc; k += 3) {
        const unsigned long long n = strtoull(argv[k], 0, 10), t = strtoull(argv[k + 1], 0, 10),
                                 i = strtoull(argv[k + 2], 0, 10);
        const GeomLayout g = geom_layout(n, t, i);
        printf("%llu %llu %llu %d\n", g.first_tri * (unsigned long long)sizeof(TriRecord),
               g.first_inst * (unsigned long long)sizeof(InstanceRecord), (unsigned long long)g.bytes, int(g.fits));
    }
}
"""


def _layouts(tmp_path, sizes):
    src, exe = tmp_path / "layout.cpp", tmp_path / "layout"
    src.write_text(PROGRAM)
    subprocess.check_call(["g++", "-std=c++17", "-I", os.path.join(ROOT, "agent-ray_b200", "csrc"), "-o", str(exe), str(src)])
    out = subprocess.check_output([str(exe)] + [str(x) for s in sizes for x in s], text=True)
    return [tuple(int(x) for x in line.split()) for line in out.splitlines()]


def test_sections_are_disjoint_and_reach_the_memory(tmp_path):
    small = [(0, 0, 0), (1, 0, 1), (2, 12, 1), (3, 1, 7), (7, 13, 5), (300, 1999, 335)]
    # 2 billion triangles, their nodes and some instances (beyond 2^32 16-byte
    # words), the most triangles that 180 GB hold, and 1 billion instances
    large = [(300_000_000, 2_000_000_000, 10_000), (1_000_000, 3_700_000_000, 1), (150_000_000, 1000, 1_000_000_000)]
    for (nodes, tris, inst), (tri_at, inst_at, total, fits) in zip(small + large, _layouts(tmp_path, small + large)):
        assert fits
        assert tri_at % 48 == 0 and inst_at % 64 == 0
        assert nodes * 80 <= tri_at < nodes * 80 + 48
        assert tri_at + tris * 48 <= inst_at < tri_at + tris * 48 + 64
        assert total == inst_at + inst * 64
    assert [f[3] for f in _layouts(tmp_path, [(1, 1 << 32, 1), (1 << 32, 1, 1), (1, 1, 1 << 32)])] == [0, 0, 0]


def test_hits_name_any_object_of_32_bits():
    # 2^30 objects and more fit the memory, and a stack entry's top bits say what
    # it is: an object index travels outside the stack.
    text = open(os.path.join(ROOT, "agent-ray_b200", "csrc", "ar_device.cuh")).read()
    body = re.sub(r"//[^\n]*", "", text[text.index("struct Traverser {"):text.index("kColdCarveout")])
    index = "m3.y"  # of the instance record being entered
    uses = [line.strip() for line in body.splitlines() if index in line]
    assert uses and not any("push" in u or "kMarker" in u for u in uses), uses
    assert not re.search(r"& *k\w*Mask", body)
