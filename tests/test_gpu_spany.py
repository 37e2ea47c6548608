"""The pseudo-spectral solver on truncated run-time-split transforms
(spany.cuh) against its general path (DNSB_FFT4=0: one Stockham transform
over the full half spectrum per field) over the lengths it accepts.

Both sum the same 64-bit products; they differ by the transforms' round-off,
a few eps log2(n) relative to the state's norm: 1e-13 over one step.
"""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _run(n, kcut, monkeypatch, general):
    from distributednavierstokes_b200 import spectral as S

    if general:
        monkeypatch.setenv("DNSB_FFT4", "0")
    s = S.spectral_setup(n=n, visc=1e-3, kcut=kcut, l=3.0)
    if general:
        monkeypatch.delenv("DNSB_FFT4")
    uh = S.specvelocity(s)
    gen = torch.Generator(device="cuda").manual_seed(7)
    v = torch.randn((3, n, n, n), generator=gen, device="cuda", dtype=torch.float64)
    S.phys_to_spec(uh, v, s)
    S.spectral_project(uh, s)
    out = [S.spec_to_phys(S.physvelocity(s), uh, s).clone(),
           S.spectral_rhs(S.specvelocity(s), uh, s).clone()]
    vmax = [S.vsummax(uh, s)]
    for _ in range(2):
        vmax.append(S.spectral_step(uh, s, 2e-3))
    s.close()
    return out + [uh], vmax


@pytest.mark.parametrize("n,kcut", [(6, None), (6, 1), (8, None), (10, 2), (12, None), (16, 5), (18, None),
                                    (20, 3), (24, None), (30, None), (32, 10), (36, 11), (40, None),
                                    (50, None), (54, 17), (60, None), (64, None), (72, 20), (80, None),
                                    (90, None), (96, 31), (100, None), (120, None), (128, None)])
def test_matches_general_path(n, kcut, monkeypatch):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    a, va = _run(n, kcut, monkeypatch, False)
    b, vb = _run(n, kcut, monkeypatch, True)
    for name, x, y in zip(("phys", "rhs", "state"), a, b):
        err = float((x - y).norm() / y.norm())
        assert err <= 1e-13, (name, err)
    for x, y in zip(va, vb):
        assert abs(x - y) <= 1e-13 * y


@pytest.mark.parametrize("n,kcut", [(192, None), (256, None), (256, 80), (384, 40)])
def test_matches_general_path_at_production_sizes(n, kcut, monkeypatch):
    """The x-kernels by warps at the splits 16 x 8 and 16 x 12 (and 8 x 12)."""
    test_matches_general_path(n, kcut, monkeypatch)
    torch.cuda.empty_cache()
