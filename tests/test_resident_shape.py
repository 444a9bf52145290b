"""The layout of a resident solve (csrc/resident_shape.hpp), on the host: on a whole B200 every
system under the row limits fits; on fewer SMs what does not fit is left to the engine."""
import os
import re
import subprocess

from conftest import ROOT

CSRC = os.path.join(ROOT, "tpt-fem_b200", "csrc")

SOURCE = r"""
#include <cstdio>
#include "resident_shape.hpp"
using namespace tptfem;
int main(int, char** v) {
  int sms, rows, dpn, na, nm, nseg;
  while (std::scanf("%d %d %d %d %d %d", &sms, &rows, &dpn, &na, &nm, &nseg) == 6) {
    const int nchunks = (rows / dpn + 31) / 32;
    const RnShape s = rn_shape(nchunks, dpn, sms, na, nm, nseg);
    std::printf("%d %d %d %d %zu %zu\n", nchunks, s.nc, s.blocks, s.w, s.smem, RN_MAX_SMEM);
  }
}
"""


def test_shapes(tmp_path):
    src, exe = tmp_path / "shape.cpp", tmp_path / "shape"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    with open(os.path.join(CSRC, "objects.hpp")) as f:
        text = f.read()
    jacobi, fsai = (int(re.search(r"%s = (\d+)" % n, text).group(1)) for n in ("RN_MAX_ROWS_JACOBI", "RN_MAX_ROWS_FSAI"))
    cases = []
    for sms in (148, 132, 74, 36, 18, 1):
        for dpn, nm in ((1, 1), (2, 3), (3, 6)):
            for rows in (dpn, 32 * dpn, 33 * dpn, 148 * 32 * dpn, fsai // 2, fsai // dpn * dpn, jacobi // dpn * dpn):
                cases.append((sms, rows, dpn, 0, 0, 0))
                if rows <= fsai:
                    cases.append((sms, rows, dpn, 256 // nm, nm, 512))  # the largest coarse space
    out = subprocess.run([str(exe)], input="\n".join(" ".join(map(str, c)) for c in cases), text=True,
                         capture_output=True, check=True).stdout.split("\n")
    refused = 0
    for c, line in zip(cases, out):
        nchunks, nc, blocks, w, smem, most = map(int, line.split())
        assert blocks <= min(c[0], 160)  # all resident at once
        assert (blocks - 1) * nc < nchunks <= blocks * nc  # every chunk has a block, every block a chunk
        assert w in (1, 2, 4, 8, 16) and w * min(nc, 16) <= 16
        assert smem >= 8 * 6 * nc * 32 * c[2] and most + 1024 <= 227 * 1024
        if c[0] >= 148:
            assert smem <= most
        refused += smem > most
    assert refused > 0
