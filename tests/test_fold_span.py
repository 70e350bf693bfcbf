"""The streamed fold's place of a row in a tile, at positions more than 2^31 apart (compiled for the host,
against Python's integers)."""
import os
import shutil
import subprocess

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "torchcompactradius_b200", "csrc")

SOURCE = r"""
#include <cstdio>
#include "tcr_fold_span.cuh"
int main() {
    long long p, t0;
    int len;
    while (std::scanf("%lld %lld %d", &p, &t0, &len) == 3) std::printf("%d\n", tcr::tile_offset(p, t0, len));
}
"""


def test_rows_far_from_the_tile(tmp_path):
    rng = np.random.default_rng(0)
    around = [0, 10, 2 ** 31 - 1, 2 ** 31, 2 ** 31 + 5, 2 ** 32, 2 ** 32 + 7, 3 * 10 ** 9, 6 * 10 ** 9, 2 ** 40]
    cases = [(p + d, t, n) for p in around for t in around for d in (-3, 0, 1, 900, 2048, 8192) for n in (1, 2048, 8192)
             if p + d >= 0]
    cases += [(int(p), int(t), 2048) for p, t in rng.integers(0, 2 ** 34, (500, 2))]
    src, exe = str(tmp_path / "span.cpp"), str(tmp_path / "span")
    with open(src, "w") as f:
        f.write(SOURCE)
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else shutil.which("g++")
    subprocess.check_call([cxx, "-std=c++17", "-x", "c++", "-I" + CSRC, "-o", exe, src])
    out = subprocess.run([exe], input="\n".join("%d %d %d" % c for c in cases), capture_output=True, text=True, check=True)
    assert [int(v) for v in out.stdout.split()] == [min(max(p - t, 0), n) for p, t, n in cases]
