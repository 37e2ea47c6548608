"""The real x-transforms by warps (k_rfftx4 / k_irfftx4, xwarp.cuh) at every
compile-time split, against the Stockham kernels (DNSB_FFT4=0) on the same input.
DNSB_XWARP=1 takes them on boxes of any size; by their own rule they run from two
blocks per SM on.

A block takes 4, 8 or 16 lines (kz) of a row, by the split, a warp 1, 2 or 4 of
them.  nz = 16 fills every block; 9 leaves warps without a line and one with half
of its lines; 25 full blocks and a last one of 1 (of 4 or 8) or 9 (of 16) lines.

Two correct FFTs of length n differ by a few eps log2(n) relative to the norm; the
Poisson solve chains six of them: 1e-13 as in test_gpu_fftany.py, and ten times
that for the velocity, whose projection takes differences of neighbouring values.
"""
import math

import pytest

torch = pytest.importorskip("torch")
import refcases as R  # noqa: E402

pytestmark = pytest.mark.gpu

SPLITS = [64, 96, 128, 192, 256, 384, 512, 768]


@pytest.fixture(scope="module")
def D():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import distributednavierstokes_b200 as dns

    return dns


def _close(a, b, tol, what):
    err = float((a - b).norm() / b.norm())
    assert err <= tol, (what, err)


def _run(D, kw, env, monkeypatch):
    monkeypatch.setenv(*env)
    s = D.setup(**kw)
    monkeypatch.delenv(env[0])
    nx, ny, nz = s.n
    gen = torch.Generator(device="cuda").manual_seed(4)
    r = torch.randn((nz, ny, nx), generator=gen, device="cuda", dtype=torch.float64)
    s.poisson["r"].copy_(r - r.mean())
    p = D.scalarfield(s)
    D.poisson(p, s)                     # a ghost-free real array in, a field with its images out
    out = [p.clone()]
    u = D.vectorfield(s)
    for c in "xyz":
        u[c][s.active(c)] = torch.randn(u[c][s.active(c)].shape, generator=gen, device="cuda",
                                        dtype=torch.float64)
    D.exchange_halo(u, s)
    psi = D.scalarfield(s)
    D.project(u, psi, s)                # a divergence in
    out += [psi.clone()] + [u[c].clone() for c in "xyz"]
    if kw["bc"][1] == "periodic":
        D.rescale_shell(u, s, 3, 1.7)   # the interior of a field in
        out += [u[c].clone() for c in "xyz"]
    s.close()
    return out


@pytest.mark.parametrize("nz", [16, 9, 25])
@pytest.mark.parametrize("bcy", ["periodic", "wall"])
@pytest.mark.parametrize("nx", SPLITS)
def test_every_split_matches_stockham(D, nx, bcy, nz, monkeypatch):
    kw = dict(n=(nx, 10, nz), bc=("periodic", bcy, "periodic"))
    if bcy == "wall":
        kw.update(lims=((0, 4.0), (-1, 1), (0, 1.0)), stretch=R.tanhstretch(1.5))
    a = _run(D, kw, ("DNSB_XWARP", "1"), monkeypatch)
    b = _run(D, kw, ("DNSB_FFT4", "0"), monkeypatch)
    for i, (x, y) in enumerate(zip(a, b)):
        _close(x, y, 1e-13 if i < 2 else 1e-12, i)


def test_full_and_short_groups_by_the_rule(D, monkeypatch):
    """A box that takes them by the rule: 192 x 90 x 27, three full groups of 8 lines
    and one of 3 per row."""
    kw = dict(n=(192, 90, 27), bc=("periodic", "periodic", "periodic"))
    a = _run(D, kw, ("DNSB_XWARP", "-1"), monkeypatch)
    b = _run(D, kw, ("DNSB_FFT4", "0"), monkeypatch)
    c = _run(D, kw, ("DNSB_XWARP", "1"), monkeypatch)
    for i, (x, y, z) in enumerate(zip(a, b, c)):
        _close(x, y, 1e-13 if i < 2 else 1e-12, i)
        assert torch.equal(x, z), i


def test_products_and_real_output(D, monkeypatch):
    """The spectral solver's general path at a side with a compile-time split of n/2
    and none of n (512): velocities out as real arrays, their products in."""
    from distributednavierstokes_b200 import spectral as S

    n, kcut = 512, 8
    out = []
    for env in (("DNSB_XWARP", "1"), ("DNSB_FFT4", "0")):
        monkeypatch.setenv(*env)
        s = S.spectral_setup(n=n, visc=1e-3, kcut=kcut, l=2 * math.pi)
        monkeypatch.delenv(env[0])
        uh = S.specvelocity(s)
        gen = torch.Generator(device="cuda").manual_seed(7)
        uh.copy_(torch.randn(uh.shape, generator=gen, device="cuda", dtype=uh.dtype))
        S.spectral_project(uh, s)
        v = S.spec_to_phys(S.physvelocity(s), uh, s)
        out.append((v[:, ::37, ::41, :].clone(), S.spectral_rhs(S.specvelocity(s), uh, s).clone()))
        del v
        s.close()
        torch.cuda.empty_cache()
    for i in range(2):
        _close(out[0][i], out[1][i], 1e-13, i)
