"""The rule that cuts the tiles of the fused 3D half steps in z, on the CPU."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "fomo.jl_b200" / "csrc"

HARNESS = r"""
#include "cuts3d.h"
extern "C" void cut(int elastic, int nt, int nz, int G, int nsm, int* out) {
  const fomo::Cuts3 c = fomo::cuts3(elastic, nt, nz, G, nsm);
  out[0] = c.tiles;
  out[1] = c.chunks;
}
// grids whose segment list would not hold their cuts, or whose cut is not one
extern "C" long long overflows() {
  long long bad = 0;
  for (int e = 0; e < 2; ++e)
    for (int nz = 1; nz <= 240; nz += nz < 16 ? 1 : 29)
      for (int G = 1; G <= 4 * fomo::kMaxGrid3; G += G < 40 ? 3 : 61)
        for (int nt = 1; nt <= 3000; nt += nt < 40 ? 3 : 97) {
          const fomo::Cuts3 c = fomo::cuts3(e, nt, nz, G, G / (2 - e) + 1);
          bad += c.tiles < 1 || c.tiles > nt || c.chunks < 1 || c.chunks > nz ||
                 nt - c.tiles + (long long)c.tiles * c.chunks > fomo::segs3_room(nt);
        }
  return bad;
}
"""


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("cuts3d")
    (d / "h.cpp").write_text(HARNESS)
    subprocess.run([cxx, "-std=c++17", "-O2", "-shared", "-fPIC", "-I", str(CSRC), "-o",
                    str(d / "h.so"), str(d / "h.cpp")], check=True)
    lib = C.CDLL(str(d / "h.so"))
    lib.overflows.restype = C.c_longlong
    return lib


def test_the_segment_list_holds_every_cut(rule):
    """Also for more CTAs than one device has."""
    assert rule.overflows() == 0


# elastic, tiles, planes, chunks: both sides of the lines, where each was measured faster
@pytest.mark.parametrize("elastic,nt,nz,chunks", [
    (0, 15, 68, 4), (0, 8, 72, 4), (0, 6, 76, 4), (0, 35, 64, 4), (0, 30, 74, 4), (0, 28, 80, 10),
    (0, 45, 67, 10), (0, 18, 58, 10), (0, 22, 48, 9), (0, 153, 209, 10), (0, 456, 108, 4),
    (1, 6, 65, 4), (1, 21, 68, 4), (1, 32, 68, 4), (1, 36, 77, 4), (1, 33, 99, 4), (1, 36, 112, 4),
    (1, 35, 142, 4), (1, 144, 147, 4), (1, 15, 94, 10), (1, 28, 80, 10), (1, 55, 128, 10),
    (1, 153, 209, 10), (1, 45, 67, 10), (1, 144, 38, 1),
])
def test_chunks(rule, elastic, nt, nz, chunks):
    out = (C.c_int * 2)()
    G = min(148 if elastic else 296, nt * nz // 16)
    rule.cut(elastic, nt, nz, G, 148, out)
    assert out[1] == chunks
    assert out[0] == (nt if chunks > 4 else min(nt, G))
