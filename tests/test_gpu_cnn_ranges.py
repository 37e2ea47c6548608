"""The closure's convolutions and weight gradients where the CTAs' ranges
start and end inside tiles and columns (odd sides, several samples, more CTAs
than tiles of a column), against the CPU oracle.  Tolerances as in
test_gpu_cnn.py: both sides round the same values to BF16 at the same points,
so only a value near a rounding boundary differs, by 2^-8."""
import math

import numpy as np
import pytest
from test_gpu_cnn import C, l2rel, maxrel  # noqa: F401

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [9, 33, 40])
def test_inference(C, n):  # noqa: F811
    closure, O = C
    cl = closure.Closure(batch=0, crop=0, nfield=n, seed=5)
    params = [(W * 3, b * 3) for W, b in closure.unflatten(cl.get_params())]
    cl.set_params(closure.flatten(params))
    params = closure.unflatten(cl.get_params())
    v = np.random.default_rng(n).standard_normal((3, n, n, n))
    got = cl.infer_cells(torch.from_numpy(v).cuda()).cpu().numpy()
    ref = O.periodic_infer(params, O.f32(v))
    assert l2rel(got, ref) <= 5e-3 and maxrel(got, ref) <= 1e-2
    cl.close()


@pytest.mark.parametrize("batch,crop", [(3, 15), (5, 12), (1, 24)])
def test_gradients(C, batch, crop):  # noqa: F811
    closure, O = C
    cl = closure.Closure(batch=batch, crop=crop, seed=17)
    params = [(W * 3, b * 3) for W, b in closure.unflatten(cl.get_params())]
    cl.set_params(closure.flatten(params))
    params = closure.unflatten(cl.get_params())
    P = crop + 8
    rng = np.random.default_rng(crop)
    x = O.f32(rng.standard_normal((batch, 3, P, P, P)))
    t = O.f32(rng.standard_normal((batch, 6, crop, crop, crop)))
    loss, g = cl.batch_grads(torch.from_numpy(x.astype(np.float32)).cuda(),
                             torch.from_numpy(t.astype(np.float32)).cuda())
    lref, gref, _ = O.loss_and_grads(params, x, t)
    assert math.isclose(loss, lref, rel_tol=1e-4)
    gd = closure.unflatten(g)
    for L in range(4):
        for k in range(2):
            assert l2rel(gd[L][k], gref[L][k]) <= 5e-3 and maxrel(gd[L][k], gref[L][k]) <= 1e-2, (L, k)
    cl.close()


def test_sides_from_two_threads(C):  # noqa: F811
    """Closures of different sides (different shared-memory needs of the same
    kernels) used at the same time from two threads give what each gives alone."""
    import threading

    closure, _ = C
    cls = [closure.Closure(batch=0, crop=0, nfield=n, seed=5) for n in (16, 64)]
    v = [torch.randn((3, n, n, n), dtype=torch.float64, device="cuda") for n in (16, 64)]
    alone = [cl.infer_cells(x).clone() for cl, x in zip(cls, v)]
    torch.cuda.synchronize()
    bad = []

    def use(i):
        try:
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                for _ in range(100):
                    got = cls[i].infer_cells(v[i])
                stream.synchronize()
                if not torch.equal(got, alone[i]):
                    bad.append(f"closure {i}: other values")
        except Exception as e:  # noqa: BLE001
            bad.append(str(e))

    threads = [threading.Thread(target=use, args=(i,)) for i in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad
    for cl in cls:
        cl.close()


def test_gradients_of_large_preactivations(C):  # noqa: F811
    """GELU's slope is 1 or 0 far from the origin, up to pre-activations whose
    square is finite in FP32: the gradients of a network with biases of +-1e15 in
    its first layer match the oracle's."""
    closure, O = C
    batch, crop = 2, 12
    cl = closure.Closure(batch=batch, crop=crop, seed=3)
    params = closure.unflatten(cl.get_params())
    W0, b0 = params[0]
    params[0] = (W0, np.where(np.arange(b0.size) % 2 == 0, 1e15, -1e15).astype(b0.dtype))
    cl.set_params(closure.flatten(params))
    params = closure.unflatten(cl.get_params())
    P = crop + 8
    rng = np.random.default_rng(1)
    x = O.f32(rng.standard_normal((batch, 3, P, P, P)))
    t = O.f32(rng.standard_normal((batch, 6, crop, crop, crop)))
    loss, g = cl.batch_grads(torch.from_numpy(x.astype(np.float32)).cuda(),
                             torch.from_numpy(t.astype(np.float32)).cuda())
    lref, gref, _ = O.loss_and_grads(params, x, t)
    assert math.isfinite(loss) and math.isclose(loss, lref, rel_tol=1e-2)
    gd = closure.unflatten(g)
    for L in range(4):
        for k in range(2):
            assert np.isfinite(gd[L][k]).all(), (L, k)
            assert l2rel(gd[L][k], gref[L][k]) <= 1e-2, (L, k)
    cl.close()
