"""The sub-tile ranges of the closure convolution: SubWalk as it stands in
distributednavierstokes_b200/csrc/cnn.cuh, compiled for the host.  The CTAs'
ranges cover every (sample, plane, sub-tile) once, differ by at most one
sub-tile, and say truthfully where a tile's planes have to be loaded (`fresh`)
and where they are used for the last time (`last`).
"""
import os
import re
import shutil
import subprocess

import pytest

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                      "distributednavierstokes_b200", "csrc", "cnn.cuh")
PROGRAM = """
#include <algorithm>
#include <cstdio>
#include <cstdlib>
using std::min;
#define __device__
#define __forceinline__ inline
struct ConvArgs { int Do, spp, sub, tpp; };
%s
int main(int, char **v) {
  ConvArgs a;
  a.Do = atoi(v[1]);
  a.spp = atoi(v[2]);
  a.sub = atoi(v[3]);
  a.tpp = (a.spp + a.sub - 1) / a.sub;
  SubWalk w;
  w.start(a, atoi(v[4]), atoi(v[5]));
  while (w.tile(a)) printf("%%d %%d %%d %%d %%d %%d %%d\\n", w.b, w.j, w.z, w.lo, w.hi, w.fresh, w.last);
}
"""


@pytest.fixture(scope="module")
def walk(tmp_path_factory):
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else shutil.which("g++")
    if not cxx:
        pytest.skip("no host compiler")
    with open(SOURCE) as f:
        struct = re.search(r"^struct SubWalk \{.*?^\};", f.read(), re.S | re.M).group(0)
    d = tmp_path_factory.mktemp("subwalk")
    (d / "w.cpp").write_text(PROGRAM % struct)
    subprocess.run([cxx, "-std=c++17", "-o", str(d / "w"), str(d / "w.cpp")], check=True)

    def run(Do, spp, sub, s0, s1):
        out = subprocess.run([str(d / "w")] + [str(v) for v in (Do, spp, sub, s0, s1)], check=True,
                             capture_output=True, text=True).stdout
        for line in out.splitlines():
            b, j, z, lo, hi, fresh, last = (int(v) for v in line.split())
            yield b, j, z, lo, hi, bool(fresh), bool(last)

    return run


@pytest.mark.parametrize("B,Do,spp,sub,grid", [
    (1, 70, 40, 3, 148),   # the last tile of a plane has one sub-tile
    (8, 38, 13, 4, 148),
    (1, 9, 2, 1, 18),      # one sub-tile a CTA
    (2, 5, 7, 4, 148),     # more CTAs than sub-tiles per column
    (1, 3, 1, 4, 3),
    (3, 1, 5, 2, 7),       # one plane: every tile loads afresh
])
def test_ranges(walk, B, Do, spp, sub, grid):
    nsub = B * Do * spp
    grid = min(grid, nsub)
    seen = []
    for cta in range(grid):
        s0, s1 = nsub * cta // grid, nsub * (cta + 1) // grid
        assert s1 - s0 in (nsub // grid, nsub // grid + 1)
        ring = []                      # planes loaded, in order
        held = 0
        for b, j, z, lo, hi, fresh, last in walk(Do, spp, sub, s0, s1):
            assert lo < hi
            ring = ([(b, j, z), (b, j, z + 1)] if fresh else ring) + [(b, j, z + 2)]
            held += 3 if fresh else 1
            # the last three planes loaded are the tile's own
            assert ring[-3:] == [(b, j, z), (b, j, z + 1), (b, j, z + 2)]
            held -= 3 if last else 1
            assert held == (0 if last else 2)
            seen += [(b, z, j * sub + s) for s in range(lo, hi)]
        assert held == 0               # every plane loaded is released
    assert sorted(seen) == [(b, z, s) for b in range(B) for z in range(Do) for s in range(spp)]
