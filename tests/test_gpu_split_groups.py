"""Edges of the split-precision group's passes: more problems than a block has
threads, pixel counts around a block's, widest legs, shapes below one row tile.
Split precision: 2e-6 + 4e-8 K of max |y|, K the longer contraction.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,Dmax,wmax", [(1, 1, 1), (1, 33, 16), (3, 129, 5), (130, 12, 4), (300, 9, 3)])
def test_split_group_sizes(ctx, n, Dmax, wmax):
    import torch
    from mpsdyn_b200 import capi
    rng = np.random.default_rng(n + Dmax)
    c = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)
    ops, inst, ys = [], [], []
    for i in range(n):
        d = int(rng.integers(1, 3))
        wl, wr = (wmax, wmax) if i == 0 else (int(rng.integers(1, wmax + 1)), int(rng.integers(1, wmax + 1)))
        Dl, Dr = (Dmax, Dmax) if i == 0 else (int(rng.integers(1, Dmax + 1)), int(rng.integers(1, Dmax + 1)))
        # memory order (slowest first): L[a, b, a'], W[c, s, b, s'], Rt[r', c, r], x[r, s, a]
        o = c(Dl, wl, Dl), c(wr, d, wl, d), c(Dr, wr, Dr), c(Dr, d, Dl)
        t = [torch.from_numpy(a).cuda() for a in o]
        y = torch.zeros(Dr * d * Dl, dtype=torch.complex128, device="cuda")
        ops.append((o, t))
        ys.append(y)
        inst.append(dict(d=d, wl=wl, wr=wr, Dl=Dl, Dr=Dr, L=t[0].data_ptr(), W=t[1].data_ptr(), Rt=t[2].data_ptr(),
                         x=t[3].data_ptr(), y=y.data_ptr()))
    torch.cuda.synchronize()
    capi.heff_matvec_grouped_ex(ctx, inst, 1, 0)
    torch.cuda.synchronize()
    for ((L, W, Rt, x), _), y in zip(ops, ys):
        want = np.einsum("abp,rsa->rsbp", L, x, optimize=True)
        want = np.einsum("csbt,rsbp->rctp", W, want, optimize=True)
        want = np.einsum("qcr,rctp->qtp", Rt, want, optimize=True).ravel()
        tol = 2e-6 + 4e-8 * max(L.shape[0], Rt.shape[0] * Rt.shape[1])
        assert np.abs(y.cpu().numpy() - want).max() <= tol * np.abs(want).max()
