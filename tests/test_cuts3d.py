"""The rule that cuts the tiles of the fused 3D half steps in z, on the CPU."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "fomo.jl_b200" / "csrc"

HARNESS = r"""
#include "cuts3d.h"
extern "C" void cut(int elastic, int nt, int nz, int G, int* out) {
  const fomo::Cuts3 c = fomo::cuts3(elastic, nt, nz, G);
  out[0] = c.tiles;
  out[1] = c.chunks;
}
// grids whose segment list would not hold their cuts, or whose cut is not one
extern "C" long long overflows() {
  long long bad = 0;
  for (int e = 0; e < 2; ++e)
    for (int nz = 1; nz <= 240; nz += nz < 70 ? 1 : 17)
      for (int G = 1; G <= 4 * fomo::kMaxGrid3; G += G < 310 ? 1 : 13)
        for (int nt = 1; nt <= 3000; nt += nt < 60 ? 1 : 37) {
          const fomo::Cuts3 c = fomo::cuts3(e, nt, nz, G);
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
