"""Edges of the Lanczos step's work split (64 rows per CTA with the basis in
registers, row ranges beyond, k up to and above 64 vectors, groups of chains of
different sizes): single-site solves of chains whose local problems have the
sizes in question reach the energy of a dense diagonalisation or of the same
solve with another split.  Energies to 1e-10, the solves' convergence.
"""
import numpy as np
import pytest

from oracle import mps_oracle as mo

pytestmark = pytest.mark.gpu


def ground(ctx, ops, L, D, **opts):
    m = ctx.mpo(ops)
    s = ctx.mps(mo.random_mps(L, 2, D, 5).sites)
    e, st = ctx.find_ground_state(m, D, s, 0.0, ctx.options(convtol=1e-11, **opts))
    m.free()
    s.free()
    return e, st


@pytest.mark.parametrize("krylov", [2, 8, 9, 17, 33, 64, 65, 120])
def test_basis_sizes_reach_the_dense_energy(ctx, krylov):
    # N up to 512 at the centre: several CTAs, every group size of basis
    # vectors, bases above 64 vectors (row ranges), restarts for the small ones
    L, D = 9, 16
    ops = mo.ising_hmpo(L, 1.0, 1.1, 0.15)
    exact = float(np.linalg.eigvalsh(mo.mpo_dense(ops))[0])
    e, st = ground(ctx, ops, L, D, max_krylov=krylov)
    assert abs(e - exact) <= 1e-10 * abs(exact)


@pytest.mark.parametrize("Ds", [(3, 40), (8, 100, 100)])
def test_groups_of_uneven_sizes(ctx, Ds):
    # chains of different bonds in one launch give the energies they have alone;
    # D = 100 has 20000 rows: row ranges instead of 64 rows per CTA
    L = 14
    ops = [mo.ising_hmpo(L, 1.0, 1.0 + 0.05 * i, 0.1) for i in range(len(Ds))]
    D = max(Ds)
    mpos = [ctx.mpo(o) for o in ops]
    alone = []
    for m, o in zip(mpos, ops):
        s = ctx.mps(mo.random_mps(L, 2, D, 7).sites)
        alone.append(ctx.find_ground_state(m, D, s, 0.0, ctx.options(convtol=1e-11))[0])
    starts = [ctx.mps(mo.random_mps(L, 2, D, 7).sites) for _ in Ds]
    es, status, _ = ctx.find_ground_state_batch(mpos, D, starts, 0.0, ctx.options(convtol=1e-11))
    assert all(st == 0 for st in status)
    for a, b in zip(es, alone):
        assert abs(a - b) <= 1e-10 * abs(b)
