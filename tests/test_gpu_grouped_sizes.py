"""Edges of the grouped product's launches: descriptors as kernel parameters (up
to 16 instances) and in device memory, the second set of launches above 192, the
small, 32- and 64-row tiles, one-site bonds and odd legs; direct and replayed
from a graph.  Complex FP64: 1e-13 of max |y| as for the single products.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def operands(rng, d, wl, wr, Dl, Dr):
    c = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)
    # memory order (slowest first): L[a, b, a'], W[c, s, b, s'], Rt[r', c, r], x[r, s, a]
    return c(Dl, wl, Dl), c(wr, d, wl, d), c(Dr, wr, Dr), c(Dr, d, Dl)


@pytest.mark.parametrize("n,Dmax", [(1, 1), (1, 16), (1, 130), (16, 40), (17, 40), (30, 300), (193, 24)])
@pytest.mark.parametrize("repeats", [0, 2])
def test_grouped_product_sizes(ctx, n, Dmax, repeats):
    import torch
    from mpsdyn_b200 import capi
    rng = np.random.default_rng(n * 1000 + Dmax)
    ops, inst, ys = [], [], []
    for i in range(n):
        d, wl, wr = int(rng.integers(1, 4)), int(rng.integers(1, 6)), int(rng.integers(1, 6))
        Dl, Dr = (Dmax, Dmax) if i == 0 else (int(rng.integers(1, Dmax + 1)), int(rng.integers(1, Dmax + 1)))
        o = operands(rng, d, wl, wr, Dl, Dr)
        t = [torch.from_numpy(a).cuda() for a in o]
        y = torch.zeros(Dr * d * Dl, dtype=torch.complex128, device="cuda")
        ops.append((o, t))
        ys.append(y)
        inst.append(dict(d=d, wl=wl, wr=wr, Dl=Dl, Dr=Dr, L=t[0].data_ptr(), W=t[1].data_ptr(), Rt=t[2].data_ptr(),
                         x=t[3].data_ptr(), y=y.data_ptr()))
    torch.cuda.synchronize()
    capi.heff_matvec_grouped(ctx, inst, repeats)
    for (o, _), y in zip(ops, ys):
        L, W, Rt, x = o
        want = np.einsum("abp,rsa->rsbp", L, x, optimize=True)
        want = np.einsum("csbt,rsbp->rctp", W, want, optimize=True)
        want = np.einsum("qcr,rctp->qtp", Rt, want, optimize=True).ravel()
        assert np.abs(y.cpu().numpy() - want).max() <= 1e-13 * max(np.abs(want).max(), 1e-300)
