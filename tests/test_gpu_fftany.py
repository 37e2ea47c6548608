"""The transform kernels with a run-time split (fftany.cuh) on every line
length they accept, against the Stockham kernels (DNSB_FFT4=0) on the same
input, and whole steps at such lengths against the oracle.

Two correct FFTs of length n differ by a few eps log2(n) relative to the
norm; the Poisson solve chains six of them, so 1e-13 (450 eps) bounds every
length here with a factor of several to spare.
"""
import math

import numpy as np
import pytest

torch = pytest.importorskip("torch")
import refcases as R  # noqa: E402

pytestmark = pytest.mark.gpu


def _smooth(n):
    for q in (2, 3, 5):
        while n % q == 0:
            n //= q
    return n == 1


LENGTHS = [n for n in range(2, 626) if _smooth(n)]


@pytest.fixture(scope="module")
def D():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import distributednavierstokes_b200 as dns

    return dns


def _solve(D, n, r):
    s = D.setup(n=n, lims=((0.0, 3.0), (0.0, 2.0), (0.0, 2.5)))
    p = D.scalarfield(s)
    s.poisson["r"].copy_(r)
    D.poisson(p, s)
    out = D.interior(p).clone()
    s.close()
    return out


@pytest.mark.parametrize("axis", ["x", "y", "z"])
def test_every_length_matches_stockham(D, axis, monkeypatch):
    gen = torch.Generator(device="cuda").manual_seed(3)
    for m in LENGTHS:
        # line counts that leave partial blocks
        n = {"x": (2 * m, 3, 9), "y": (10, m, 9), "z": (10, 9, m)}[axis]
        r = torch.randn((n[2], n[1], n[0]), generator=gen, device="cuda", dtype=torch.float64)
        r -= r.mean()
        a = _solve(D, n, r)
        monkeypatch.setenv("DNSB_FFT4", "0")
        b = _solve(D, n, r)
        monkeypatch.delenv("DNSB_FFT4")
        err = float((a - b).norm() / b.norm())
        assert err <= 1e-13, (axis, m, err)


@pytest.mark.parametrize("n,bcy,yd", [((50, 45, 27), "periodic", "explicit"),
                                      ((36, 15, 25), "periodic", "explicit"),
                                      ((90, 41, 54), "wall", "implicit"),
                                      ((250, 21, 15), "wall", "explicit")])
def test_one_step_odd_lengths(D, oracle_mod, n, bcy, yd):
    kw = R.case_kwargs(bcy, n=n, visc=0.01, ydiffusion=yd)
    so, sd = oracle_mod.Setup(**kw), D.setup(**kw)
    v = R.random_values(so)
    u = so.vectorfield()
    for c in "xyz":
        u[c][so.active(c)] = 0.3 * v[c]
    so.exchange_halo(u)
    so.project(u, so.scalarfield())
    ud = D.VectorField(**{c: torch.from_numpy(u[c].copy()).cuda() for c in "xyz"})
    p, q, d = so.scalarfield(), so.vectorfield(), so.scalarfield()
    so.step(u, p, q, d if yd == "implicit" else p, 1e-3)
    pd, qd = D.scalarfield(sd), D.vectorfield(sd)
    D.step(ud, pd, qd, D.scalarfield(sd) if yd == "implicit" else None, sd, 1e-3)
    for c in "xyz":
        a = ud[c].cpu().numpy()
        assert np.max(np.abs(a - u[c])) <= 1e-12 * np.max(np.abs(u[c])), c
    assert math.isfinite(float(pd.abs().max()))
    assert D.maxdiv(ud, sd) < 1e-10
    sd.close()
