"""The sub-tile ranges of the closure convolution (SubWalk in
distributednavierstokes_b200/csrc/cnn.cuh), mirrored on the host: the CTAs'
ranges cover every (sample, plane, sub-tile) once, differ by at most one
sub-tile, and say truthfully where a tile's planes have to be loaded (`fresh`)
and where they are used for the last time (`last`).
"""
import pytest


def walk(B, Do, spp, sub, s0, s1):
    tpp = -(-spp // sub)
    b, r = divmod(s0, spp * Do)
    j, r = divmod(r, sub * Do)
    n = min(sub, spp - j * sub)
    z, lo = divmod(r, n)
    z, left, first = z - 1, s1 - s0, True
    while left > 0:
        z += 1
        if z == Do:
            z, j = 0, j + 1
            if j == tpp:
                j, b = 0, b + 1
            n = min(sub, spp - j * sub)
        if not first:
            lo = 0
        hi = min(n, lo + left)
        left -= hi - lo
        yield b, j, z, lo, hi, first or z == 0, left == 0 or z == Do - 1
        first = False


@pytest.mark.parametrize("B,Do,spp,sub,grid", [
    (1, 70, 40, 3, 148),   # the last tile of a plane has one sub-tile
    (8, 38, 13, 4, 148),
    (1, 9, 2, 1, 18),      # one sub-tile a CTA
    (2, 5, 7, 4, 148),     # more CTAs than sub-tiles per column
    (1, 3, 1, 4, 3),
    (3, 1, 5, 2, 7),       # one plane: every tile loads afresh
])
def test_ranges(B, Do, spp, sub, grid):
    nsub = B * Do * spp
    grid = min(grid, nsub)
    seen = []
    for cta in range(grid):
        s0, s1 = nsub * cta // grid, nsub * (cta + 1) // grid
        assert s1 - s0 in (nsub // grid, nsub // grid + 1)
        ring = []                      # planes loaded, in order
        held = 0
        for b, j, z, lo, hi, fresh, last in walk(B, Do, spp, sub, s0, s1):
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
