"""Edges of the cluster QR (one CTA per 16 columns, rows in registers by 32,
the one-CTA form up to 32 x 16, the switch to the global-memory kernels)
against LAPACK, whose conventions it keeps, and the strided site form through
the gauge moves.  Tolerances as for the other QR tests: 1e-13 sqrt(m) on the
product and the orthonormality, 1e-11 on the factors themselves.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rand_c(rng, shape):
    return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)


@pytest.mark.parametrize("m,n", [(1, 1), (1, 16), (32, 16), (33, 16), (32, 17), (31, 15), (64, 33), (65, 48), (128, 16),
                                 (129, 31), (256, 129), (257, 128), (511, 255), (512, 256), (512, 257), (513, 64), (17, 256)])
def test_qr_sizes_match_lapack(ctx, m, n):
    rng = np.random.default_rng(1000 * m + n)
    A = rand_c(rng, (m, n))
    Q, R = ctx.qr(A)
    Qn, Rn = np.linalg.qr(A, mode="reduced")
    K = min(m, n)
    assert np.abs(Q @ R - A).max() < 1e-13 * np.abs(A).max() * max(m, n) ** 0.5
    assert np.abs(Q.conj().T @ Q - np.eye(K)).max() < 1e-13 * max(m, n) ** 0.5
    assert np.abs(R - Rn).max() < 1e-11 * np.abs(Rn).max() and np.abs(Q - Qn).max() < 1e-11


@pytest.mark.parametrize("m,n", [(20, 12), (300, 40)])
def test_qr_columns_without_representable_squares(ctx, m, n):
    # columns whose squares underflow or overflow, zero columns, a zero block, a -0.0 pivot
    rng = np.random.default_rng(m)
    A = rand_c(rng, (m, n))
    A[:, 1] *= 1e-170
    A[:, 2] *= 1e160
    A[:, 3] = 0.0
    A[:, n - 3:] = 0.0
    A[5:, 4] = 0.0
    A[4, 4] = complex(-0.0, -3e-200)
    Q, R = ctx.qr(A)
    Qn, Rn = np.linalg.qr(A, mode="reduced")
    assert np.all(np.isfinite(Q)) and np.all(np.isfinite(R))
    assert np.abs(Q.conj().T @ Q - np.eye(n)).max() < 1e-13 * m ** 0.5
    # column by column: each is reproduced at its own scale
    for j in range(n):
        scale = max(np.abs(A[:, j]).max(), 1e-300)
        assert np.abs((Q @ (R[:, j] / scale)) - A[:, j] / scale).max() < 1e-12


@pytest.mark.parametrize("d,Dl,Dr", [(2, 128, 128), (2, 100, 37), (3, 7, 30), (2, 1, 2), (2, 200, 120)])
def test_gauge_moves_through_strided_views(ctx, d, Dl, Dr):
    # a three-site chain whose middle site is moved in both directions: the
    # state is unchanged and the moved site is an isometry
    rng = np.random.default_rng(d * Dl + Dr)
    a, b = min(Dl, d), min(Dr, d)
    sites = [rand_c(rng, (d, 1, a)), rand_c(rng, (d, a, b)), rand_c(rng, (d, b, 1))]
    if Dl > d or Dr > d:  # wide bonds: only the middle site's shape matters
        sites = [rand_c(rng, (d, 1, Dl)), rand_c(rng, (d, Dl, Dr)), rand_c(rng, (d, Dr, 1))]

    def amplitude(s):
        return np.einsum("sab,tbc,ucd->stu", *s)

    ref = amplitude(sites)
    for direction in "RL":
        psi = ctx.mps(sites)
        psi.gauge(direction)  # normalises: the amplitudes up to the norm
        got, _ = psi.download()
        psi.free()
        amp = amplitude(got)
        amp = amp * (np.vdot(amp, ref) / np.vdot(amp, amp))
        assert np.abs(amp - ref).max() < 1e-11 * np.abs(ref).max()
        A = got[1]
        g = np.einsum("sab,sac->bc", A.conj(), A) if direction == "R" else np.einsum("sab,scb->ac", A, A.conj())
        assert np.abs(g - np.eye(g.shape[0])).max() < 1e-12
