"""Compiles a few lines of host C++ against the library's own box-table header
(isothermal_mhd_b200/csrc/imhd_table.h), so that tests can ask it for a box's
column lengths and block counts without a GPU."""
import os
import subprocess

from isothermal_mhd_b200 import build

SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include "imhd_table.h"

int main(int argc, char** argv) {
    for (int a = 1; a + 3 <= argc; a += 3) {
        for (size_t esz : {size_t(4), size_t(8)}) {
            imhd::BoxRec r;
            imhd::init_rec(r, atoi(argv[a]), atoi(argv[a + 1]), atoi(argv[a + 2]), 1, 2, 0, 1.0, 0.4, 0.0, 0.0);
            imhd::one_box_segments(r, esz);
            std::printf("%d %d\n", 1 << r.segs, 1 << r.segzs);
        }
    }
}
"""


def run(source, args, workdir):
    """Output lines of a host program built from `source`."""
    src, exe = os.path.join(workdir, "probe.cpp"), os.path.join(workdir, "probe")
    with open(src, "w") as f:
        f.write(source)
    cuda = os.path.join(os.path.dirname(os.path.dirname(build.nvcc())), "include")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-I", cuda, "-I", build.CSRC, src, "-o", exe])
    return subprocess.run([exe] + [str(v) for v in args], check=True, capture_output=True, text=True).stdout.split("\n")[:-1]


def column_lengths(boxes, workdir):
    """Per box {32: (sweep, z), 64: (sweep, z)}: cells per thread of a single box's y / z sweeps and z-column kernels."""
    lines = run(SOURCE, [v for n in boxes for v in n], workdir)
    pairs = [tuple(int(v) for v in s.split()) for s in lines]
    return [{32: pairs[2 * i], 64: pairs[2 * i + 1]} for i in range(len(boxes))]
