"""Tile and cluster shapes of the FP64 contractions at their edges: 64-row tiles by
themselves and in clusters of 2 and 4, the smallest K shares, MPO legs on the tensor
pipe with every remainder and legs whose tables leave the scalar form.  Complex FP64:
1e-13 of max |y| (sums of at most 2,000 terms).
"""
import numpy as np
import pytest

from oracle import mps_oracle as mo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,wl,wr,Dl,Dr", [
    (1, 2, 3, 3, 256, 256),   # 64 rows, clusters of 4
    (1, 2, 3, 5, 251, 253),   # the same, ragged
    (8, 2, 5, 5, 128, 128),   # 64 rows, clusters of 2; 64-row legs
    (8, 2, 5, 4, 127, 113),
    (16, 2, 5, 5, 130, 126),  # 64 rows alone
    (1, 2, 2, 2, 31, 33),     # K = 66: no cluster with a share under two slabs
    (1, 2, 1, 1, 17, 200),    # one bond leg
    (2, 3, 7, 6, 40, 45),     # 18 and 21 legs: every remainder of 8 and 4
    (1, 3, 10, 9, 30, 20),
    (1, 1, 32, 30, 20, 18),
])
def test_contraction_tiles(ctx, n, d, wl, wr, Dl, Dr):
    import torch
    from mpsdyn_b200 import capi
    rng = np.random.default_rng(n + 10 * wl + Dl)
    c = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)
    # memory order (slowest first): L[a, b, a'], W[c, s, b, s'], Rt[r', c, r], x[r, s, a]
    ops = [(c(Dl, wl, Dl), c(wr, d, wl, d), c(Dr, wr, Dr), c(Dr, d, Dl)) for _ in range(n)]
    t = [[torch.from_numpy(a).cuda() for a in o] for o in ops]
    ys = [torch.zeros(Dr * d * Dl, dtype=torch.complex128, device="cuda") for _ in range(n)]
    torch.cuda.synchronize()
    capi.heff_matvec_grouped(ctx, [dict(d=d, wl=wl, wr=wr, Dl=Dl, Dr=Dr, L=a.data_ptr(), W=b.data_ptr(),
                                        Rt=r.data_ptr(), x=x.data_ptr(), y=y.data_ptr())
                                   for (a, b, r, x), y in zip(t, ys)], 0)
    for (L, W, Rt, x), y in zip(ops, ys):
        want = np.einsum("abp,rsa->rsbp", L, x, optimize=True)
        want = np.einsum("csbt,rsbp->rctp", W, want, optimize=True)
        want = np.einsum("qcr,rctp->qtp", Rt, want, optimize=True).ravel()
        assert np.abs(y.cpu().numpy() - want).max() <= 1e-13 * np.abs(want).max()


# legs whose tables just fit behind the 32-row tile (39 x 39), and that leave the scalar form
@pytest.mark.parametrize("d,w", [(3, 13), (3, 14), (4, 16), (2, 32)])
def test_wide_legs(ctx, d, w):
    rng = np.random.default_rng(100 * d + w)
    c = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)
    Dl, Dr = 20, 23
    L, W, R = c(Dl, w, Dl), c(d, w, d, w), c(Dr, w, Dr)
    pairs = [(ctx.heff_matvec(L, W, R, x, 0.3), mo.heff_matvec(L, W, R, x, 0.3)) for x in [c(d * Dl * Dr)]]
    ket, bra = c(d, Dl, Dr), c(d, Dl, Dr)
    pairs += [(ctx.env_left(L, ket, W, bra), mo.env_left(L, ket, W, bra)),
              (ctx.env_right(R, ket, W, bra), mo.env_right(R, ket, W, bra))]
    for got, want in pairs:
        assert np.abs(got - want).max() <= 1e-13 * np.abs(want).max()
