"""Edges of the cluster QR's 8-column tiles: one and two tiles per CTA, panels with
fewer than 8 reflectors, row counts around 16 and around the register plans (64,
128, 256, 512 rows), zero and dependent columns in the middle of a panel.
Tolerances as for the other QR tests.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(33, 1), (33, 8), (34, 9), (47, 23), (49, 24), (64, 128), (65, 127), (128, 120), (129, 7),
                                 (255, 121), (256, 128), (257, 128), (256, 129), (264, 136), (40, 250), (496, 129),
                                 (511, 8), (512, 249)])
def test_qr_tile_edges_match_lapack(ctx, m, n):
    rng = np.random.default_rng(7 * m + n)
    A = rng.standard_normal((m, n)) + 1j * rng.standard_normal((m, n))
    Q, R = ctx.qr(A)
    Qn, Rn = np.linalg.qr(A, mode="reduced")
    K = min(m, n)
    assert np.abs(Q @ R - A).max() < 1e-13 * np.abs(A).max() * max(m, n) ** 0.5
    assert np.abs(Q.conj().T @ Q - np.eye(K)).max() < 1e-13 * max(m, n) ** 0.5
    assert np.abs(R - Rn).max() < 1e-11 * np.abs(Rn).max() and np.abs(Q - Qn).max() < 1e-11


@pytest.mark.parametrize("m,n,zero", [(70, 30, 11), (300, 140, 131), (36, 20, 15)])
def test_qr_degenerate_columns(ctx, m, n, zero):
    rng = np.random.default_rng(m)
    A = rng.standard_normal((m, n)) + 1j * rng.standard_normal((m, n))
    A[:, zero] = 0.0
    A[:, zero + 1] = A[:, 0] * (2 - 1j)
    A[:, zero + 2] *= 1e-170
    A[:, 3] *= 1e165
    Q, R = ctx.qr(A)
    assert np.all(np.isfinite(Q)) and np.all(np.isfinite(R))
    assert np.abs(Q.conj().T @ Q - np.eye(n)).max() < 1e-13 * m ** 0.5
    for j in range(n):  # each column at its own scale
        scale = max(np.abs(A[:, j]).max(), 1e-300)
        assert np.abs((Q @ (R[:, j] / scale)) - A[:, j] / scale).max() < 1e-12


@pytest.mark.parametrize("m,n", [(32, 8), (40, 8), (70, 1), (300, 5)])
def test_qr_of_nan_is_nan(ctx, m, n):
    """A column of NaN below a finite pivot is no column of zeros for the cluster forms: R shows it."""
    A = np.random.default_rng(m).standard_normal((m, n)) + 0j
    A[1:, 0] = complex(np.nan, np.nan)
    Q, R = ctx.qr(A)
    assert np.isnan(R[0, 0]) and np.isnan(Q[:, 0]).any()
