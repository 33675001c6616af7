"""Edges of the block Jacobi SVD (one CTA up to 16 columns, pairs of blocks of 8
on a cluster, on the grid above 256 columns, the global-memory form for long
columns) against LAPACK: Schmidt values and SVD cuts of chains whose central
bonds have the size in question.  Jacobi values carry a few ulps per sweep of
the largest one: 1e-12.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def chain(L, d, D, seed):
    rng = np.random.default_rng(seed)
    bond = [int(min(D, d ** min(k, L - k))) for k in range(L + 1)]
    return [(rng.standard_normal((d, a, r)) + 1j * rng.standard_normal((d, a, r))) / np.sqrt(2.0 * d * a)
            for a, r in zip(bond, bond[1:])]


def cut_left(sites, D):
    """SVD cuts to D from the right end, the factor passed to the left."""
    out, carry, dropped = [], np.eye(1), 0.0
    for A in reversed(sites):
        A = np.einsum("sar,rq->saq", A, carry)
        d, a, q = A.shape
        U, s, Vh = np.linalg.svd(A.transpose(1, 0, 2).reshape(a, d * q), full_matrices=False)
        k = min(D, len(s))
        dropped += np.sum(s[k:] ** 2)
        out.append(Vh[:k].reshape(k, d, q).transpose(1, 0, 2))
        carry = U[:, :k] * s[:k]
    return out[::-1], carry[0, 0], dropped, s


def overlap(x, y):
    e = np.ones((1, 1))
    for a, b in zip(x, y):
        e = np.einsum("ab,sac,sbd->cd", e, a.conj(), b, optimize=True)
    return e[0, 0]


def schmidt(sites, pos):
    left, _, _, _ = cut_left(sites, 1 << 30)  # right-canonical, then the left part's factor
    R = np.eye(1)
    for A in left[:pos]:
        A = np.einsum("ab,sbr->sar", R, A)
        R = np.linalg.qr(A.reshape(-1, A.shape[2]))[1]
    s = np.linalg.svd(R, compute_uv=False) ** 2
    return s / s.sum()


@pytest.mark.parametrize("d,L,D", [(2, 2, 2), (2, 8, 15), (2, 9, 16), (2, 10, 17), (2, 12, 31), (2, 12, 33), (2, 12, 64),
                                   (2, 14, 100), (3, 10, 129), (2, 16, 256), (2, 18, 257), (3, 12, 300)])
def test_schmidt_values_match_lapack(ctx, d, L, D):
    sites = chain(L, d, D, D)
    psi = ctx.mps(sites)
    got = np.sort(ctx.schmidt_values(psi, L // 2))[::-1]
    psi.free()
    want = np.sort(schmidt(sites, L // 2))[::-1]
    n = min(len(got), len(want))
    assert np.abs(got[:n] - want[:n]).max() < 1e-12 * want[0]
    assert np.all(got[n:] < 1e-24)


@pytest.mark.parametrize("d,L,D,cut", [(2, 6, 8, 3), (2, 9, 16, 7), (2, 10, 24, 20), (2, 12, 64, 16), (3, 8, 81, 40),
                                       (2, 16, 200, 100), (2, 18, 280, 64), (3, 12, 300, 90)])
def test_cuts_match_lapack(ctx, d, L, D, cut):
    sites = chain(L, d, D, D + cut)
    psi = ctx.mps(sites)
    phi, discarded = psi.approximate(cut)
    got, norm = phi.download()
    psi.free()
    phi.free()
    want, wnorm, dropped, _ = cut_left(sites, cut)
    assert abs(norm / abs(wnorm) - 1) < 1e-12
    assert abs(discarded - dropped) < 1e-12 * max(dropped, abs(wnorm) ** 2)
    assert abs(abs(overlap(got, want)) - 1) < 1e-11
    assert abs(overlap(got, got) - 1) < 1e-11


@pytest.mark.parametrize("D", [2, 7, 16, 24, 40])
def test_parallel_columns_settle(ctx, D):
    """Columns parallel to the first one shrink by a rounding error a sweep, to zero through values whose squares
    underflow: the last site's matrix of rank 1 with columns of falling size, cut to all of them."""
    rs = np.random.RandomState(D)
    d = max(2, D)
    A = rs.standard_normal((d, 1, D)) + 1j * rs.standard_normal((d, 1, D))
    B = np.zeros((d, D, 1), dtype=complex)
    B[0, :, 0] = rs.standard_normal(D) * 10.0 ** -np.linspace(0, 17, D)
    cut, disc = ctx.mps([np.asfortranarray(A), np.asfortranarray(B)]).approximate(D)
    assert abs(np.max(ctx.schmidt_values(cut, 1)) - 1.0) < 1e-12 and disc < 1e-24


@pytest.mark.parametrize("D", [12, 24, 40])
def test_doubly_graded_matrix_settles(ctx, D):
    """Rows and columns that both fall off by 1e-3 an index: pairs of columns of 1e-80, whose squares' product
    underflows."""
    rs = np.random.RandomState(D)
    g = 10.0 ** -(np.arange(D) * 100.0 / D)
    M = g[:, None] * (rs.standard_normal((D, D)) + 1j * rs.standard_normal((D, D))) * g
    A = rs.standard_normal((D, 1, D)) + 1j * rs.standard_normal((D, 1, D))
    cut, disc = ctx.mps([np.asfortranarray(A), np.asfortranarray(M.reshape(D, D, 1))]).approximate(D)
    s = np.linalg.svd(A[:, 0] @ M.T, compute_uv=False)
    assert abs(np.max(ctx.schmidt_values(cut, 1)) - s[0] ** 2 / np.sum(s**2)) < 1e-12 and disc < 1e-24


@pytest.mark.parametrize("low", [1e-150, 1e-155, 1e-160])
@pytest.mark.parametrize("D", [12, 20, 40, 300])
def test_tiny_columns_leave_the_large_ones_alone(ctx, D, low):
    """A matrix whose first two rows hold its two largest values and the others are of `low`, where squares of products
    underflow: the weight that a cut to one value discards is the second value's square, |det| / s_1 of the first two rows."""
    rs = np.random.RandomState(D)
    G = rs.standard_normal((D, D)) + 1j * rs.standard_normal((D, D))
    c = np.full(D, low) * 10.0 ** rs.uniform(-5, 5, D)
    c[:2] = 1.0, 1.7e-6
    U = np.linalg.qr(rs.standard_normal((D, D)) + 1j * rs.standard_normal((D, D)))[0]
    psi = ctx.mps([np.asfortranarray(U.reshape(D, 1, D)), np.asfortranarray((c[:, None] * G).reshape(D, D, 1))])
    phi, discarded = psi.approximate(1)
    psi.free()
    phi.free()
    R = np.linalg.qr(G[:2].conj().T)[1]
    s1 = np.linalg.norm(c[:2, None] * R.conj().T, 2)
    assert abs(discarded / (c[1] * abs(R[0, 0] * R[1, 1]) / s1) ** 2 - 1.0) < 1e-12


@pytest.mark.parametrize("scale", [1e-76, 1e-77])
@pytest.mark.parametrize("D", [12, 20, 40, 300])
def test_values_of_tiny_matrices(ctx, D, scale):
    """A matrix whose columns are all so small that squares of their products underflow: a cut discards the same share
    of the weight as at scale one (pairs left alone, with products below 2e-162, are orthogonal to 1e-8 there)."""
    rs = np.random.RandomState(D)
    cut = min(D // 2, 20)
    G = rs.standard_normal((D, D)) + 1j * rs.standard_normal((D, D))
    U = np.linalg.qr(rs.standard_normal((D, D)) + 1j * rs.standard_normal((D, D)))[0]
    psi = ctx.mps([np.asfortranarray(U.reshape(D, 1, D)), np.asfortranarray((scale * G).reshape(D, D, 1))])
    phi, discarded = psi.approximate(cut)
    psi.free()
    phi.free()
    s = np.linalg.svd(G, compute_uv=False)
    assert abs(discarded / scale / scale / np.sum(s[cut:] ** 2) - 1.0) < 1e-12


@pytest.mark.parametrize("order", ["mixed", "rising"])
@pytest.mark.parametrize("L,D,low", [(12, 64, 60), (14, 128, 100), (16, 256, 60)])
def test_unsorted_gradings_settle(ctx, L, D, low, order):
    """A bond whose coefficients fall over many orders in no order, or rise: Schmidt values and a cut settle."""
    rs = np.random.RandomState(5)
    s = 10.0 ** -np.linspace(0, low, D)
    s = s[rs.permutation(D)] if order == "mixed" else s[::-1]
    bond = [min(D, 2 ** min(k, L - k)) for k in range(L + 1)]
    sites = []
    for k, (a, r) in enumerate(zip(bond, bond[1:])):
        if k < L // 2:
            A = np.linalg.qr(rs.standard_normal((2 * a, r)) + 1j * rs.standard_normal((2 * a, r)))[0].reshape(2, a, r)
        else:
            A = np.linalg.qr(rs.standard_normal((2 * r, a)) + 1j * rs.standard_normal((2 * r, a)))[0]
            A = A.conj().T.reshape(a, 2, r).transpose(1, 0, 2)
        sites.append(np.asfortranarray(s[None, :, None] * A if k == L // 2 else A))
    psi = ctx.mps(sites)
    want = np.sort(s**2 / np.sum(s**2))[::-1]
    phi, discarded = psi.approximate(D // 2)
    for state in (psi, phi):
        got = np.sort(ctx.schmidt_values(state, L // 2))[::-1][: D // 2]
        assert np.max(np.abs(got - want[: D // 2])) < 1e-12
        state.free()
    assert 0.0 <= discarded < 1e-24
