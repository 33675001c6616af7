"""Measurements whose left and right chains run side by side: Schmidt values of every bond and local
observables of every site, against the dense state, at the ends of a chain, at bonds of one and of odd size,
and for states where the product of the two factors is left to the sweep (a zero product, norms near the
limits of the type)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SX = np.array([[0, 1], [1, 0]], dtype=complex)


def sites_of(L, d, bonds, seed):
    rs = np.random.RandomState(seed)
    bonds = [1] + list(bonds) + [1]
    return [np.asfortranarray(rs.standard_normal((d, a, r)) + 1j * rs.standard_normal((d, a, r))) / np.sqrt(d * a)
            for a, r in zip(bonds, bonds[1:])]


def dense(sites):
    v = np.ones((1, 1), dtype=complex)
    for A in sites:
        v = np.einsum("xa,sar->xsr", v, A).reshape(-1, A.shape[2])
    return v.reshape([A.shape[0] for A in sites])


def schmidt(sites, pos):
    v = dense(sites)
    s = np.linalg.svd(v.reshape(int(np.prod(v.shape[:pos])), -1), compute_uv=False)
    return s**2 / np.sum(s**2)


def check_schmidt(got, want, tol):
    got = np.sort(np.asarray(got))[::-1]
    assert np.all(np.isfinite(got)) and abs(got.sum() - 1.0) < tol
    n = min(len(got), len(want))
    assert np.max(np.abs(got[:n] - want[:n])) < tol
    assert np.all(got[n:] < tol) and np.all(want[n:] < tol)


# a factorisation and a product per site lose a few units of rounding of the norm: 12 sites of at most 20 x 2
# values stay below 1e-12
TOL = 1e-12


@pytest.mark.parametrize("L,d,bonds", [
    (2, 2, [2]), (3, 2, [1, 2]), (7, 2, [2, 3, 7, 5, 3, 2]), (8, 2, [2, 4, 8, 16, 8, 4, 2]),
    (6, 3, [3, 9, 20, 9, 3]), (10, 2, [1] * 9), (9, 2, [2, 4, 1, 2, 4, 5, 4, 2]), (2, 18, [17]), (3, 20, [1, 20]),
    (10, 2, [2, 4, 8, 16, 17, 13, 8, 4, 2]), (10, 2, [2, 4, 8, 16, 32, 16, 1, 2, 2])])
def test_schmidt_values_of_every_bond(ctx, L, d, bonds):
    sites = sites_of(L, d, bonds, 7)
    psi = ctx.mps(sites)
    for pos in range(1, L):
        check_schmidt(ctx.schmidt_values(psi, pos), schmidt(sites, pos), TOL)
    check_schmidt(ctx.schmidt_values(psi, 0), schmidt(sites, L // 2), TOL)


def test_bonds_above_the_rank(ctx):
    """Sites whose bonds carry a rank of 2 padded to 24: the factors' rows fall off by a rounding error per site."""
    L, d, D, r = 40, 2, 24, 2
    core = sites_of(L, d, [r] * (L - 1), 17)
    rs = np.random.RandomState(19)
    mix = [np.linalg.qr(rs.standard_normal((D, D)) + 1j * rs.standard_normal((D, D)))[0] for _ in range(L - 1)]
    big = []
    for k, A in enumerate(core):
        if k:
            A = np.einsum("ba,sar->sbr", mix[k - 1][:, :r], A)
        if k < L - 1:
            A = np.einsum("sar,br->sab", A, mix[k][:, :r].conj())
        big.append(np.asfortranarray(A))
    for pos in (1, 13, 20, 39):
        # the left and right halves' Gram matrices in the bond of rank 2
        G, H = np.ones((1, 1)), np.ones((1, 1))
        for A in core[:pos]:
            G = np.einsum("ab,sar,sbt->rt", G, A.conj(), A)
        for A in core[pos:][::-1]:
            H = np.einsum("ab,sra,stb->rt", H, A, A.conj())
        lam = np.sort(np.linalg.eigvals(G @ H).real)[::-1]
        check_schmidt(ctx.schmidt_values(ctx.mps(big), pos), lam / lam.sum(), 4 * TOL)


@pytest.mark.parametrize("scale", [1e145, 1e-145])
def test_norms_near_the_limits_go_to_the_sweep(ctx, scale):
    sites = sites_of(4, 5, [5, 20, 5], 3)
    want = schmidt(sites, 2)
    sites[2] = sites[2] * scale
    check_schmidt(ctx.schmidt_values(ctx.mps(sites), 2), want, TOL)


def test_orthogonal_halves_go_to_the_sweep(ctx):
    """A product of norm 1e-6 of its factors': the sweep carries the left factor into the next site, where nothing of the
    large part meets it, so that no accuracy is lost."""
    sites = sites_of(2, 20, [20], 5)
    sites[0][:, :, 10:] = 0.0
    sites[1][:, :10, :] *= 1e-6
    check_schmidt(ctx.schmidt_values(ctx.mps(sites), 1), schmidt(sites, 1), TOL)


@pytest.mark.parametrize("L,d,bonds", [(1, 2, []), (2, 2, [2]), (3, 2, [2, 2]), (7, 2, [2, 3, 7, 5, 3, 2]), (6, 3, [3, 9, 20, 9, 3])])
def test_local_observables_of_every_site(ctx, L, d, bonds):
    sites = sites_of(L, d, bonds, 11)
    op = SX if d == 2 else np.diag([1.0, -0.5, 0.25]).astype(complex) + np.eye(3, k=1) + np.eye(3, k=-1)
    v = dense(sites)
    got = ctx.expectation_local(ctx.mps(sites), op)
    for k in range(L):
        w = np.moveaxis(np.tensordot(op, v, axes=(1, k)), 0, k)
        assert abs(got[k] - (np.vdot(v, w) / np.vdot(v, v)).real) < TOL


@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("D", [12, 20, 40])
def test_graded_schmidt_values(ctx, D, split):
    """Coefficients that fall evenly from 1 to 1e-40, on one site or split over both: every one to a few ulps of itself
    (a factorisation, a product and the rotations keep the columns' scales)."""
    rs = np.random.RandomState(D)
    U, V = (np.linalg.qr(rs.standard_normal((D, D)) + 1j * rs.standard_normal((D, D)))[0] for _ in range(2))
    s = 10.0 ** -np.linspace(0, 40, D)
    left, right = (np.sqrt(s), np.sqrt(s)) if split else (np.ones(D), s)
    psi = ctx.mps([np.asfortranarray((U * left).reshape(D, 1, D)), np.asfortranarray((right[:, None] * V).T.reshape(D, D, 1))])
    got = np.sort(ctx.schmidt_values(psi, 1))
    psi.free()
    want = np.sort(s**2 / np.sum(s**2))
    assert np.max(np.abs(got / want - 1.0)) < TOL


@pytest.mark.parametrize("flip", [False, True])
@pytest.mark.parametrize("D", [24, 64])
def test_schmidt_values_after_a_quench(ctx, D, flip):
    """Short evolution from a product state at bonds far above its rank: factors whose rows fall off by tens of orders,
    further on one side of the bond than on the other; every bond of the chain and of its mirror image settles, with the
    Schmidt values of the two halves' Gram matrices."""
    L = 24
    U = ctx.mpo_ising_evolution(L, 1.0, 1.3, 0.1, 0.01, False)
    psi, o = ctx.mps_product(L, 2, 1), ctx.options(convtol=1e-10)
    for _ in range(8):
        aux = psi.copy()
        ctx.optimize(U, aux, psi, D, o)
        aux.free()
    sites = psi.download()[0]
    if flip:
        sites = [np.asfortranarray(np.transpose(A, (0, 2, 1))) for A in sites[::-1]]
    state = ctx.mps(sites)
    for pos in range(1, L):
        G, H = np.ones((1, 1)), np.ones((1, 1))
        for A in sites[:pos]:
            G = np.einsum("ab,sar,sbt->rt", G, A.conj(), A, optimize=True)
        for A in sites[pos:][::-1]:
            H = np.einsum("ab,sra,stb->rt", H, A, A.conj(), optimize=True)
        lam = np.sort(np.linalg.eigvals(G @ H).real)[::-1]
        check_schmidt(ctx.schmidt_values(state, pos), lam / lam.sum(), 4 * TOL)
    for x in (U, psi, state):
        x.free()
