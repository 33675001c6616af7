"""Kernels launched before their predecessor has ended give the bits of separately
synchronised ones: gauge moves and products of bonds on both sides of the grid size
(74 blocks) from which kernels launch as usual.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [1, 9, 16, 40, 100])
def test_chained_kernels_match_synchronised_ones(ctx, D):
    psi = ctx.mps_random_state(10, 2, D, 7)
    a, b = psi.copy(), psi.copy()
    for direction in "RLRL":
        a.gauge(direction)
    for direction in "RLRL":
        ctx.synchronize()
        b.gauge(direction)
        ctx.synchronize()
    for x, y in zip(a.download()[0], b.download()[0]):
        assert np.array_equal(x, y)
    one = ctx.contract(a, None, psi)
    for _ in range(5):
        assert ctx.contract(a, None, psi) == one
    for p in (psi, a, b):
        p.free()
