"""FP64 products of a residual (X, I4, ring, ladders) against the oracle, over the warp tiles the
plan picks: 4-row tiles on the smallest lattices, 8-row tiles, and several row tiles a warp.

Both sides sum in FP64 in different orders: blocks agree to 1e-12 of the largest entry, as in the
other residual comparisons (1e-11 for the complex interaction)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nmax,A,rho,snm", [
    (1, 2, 0.16, False),    # one hole pair: N = 1, K = 1 blocks
    (1, 14, 0.08, False),
    (1, 38, 0.16, False),   # more holes than particles
    (1, 4, 0.16, True),     # complex
    (2, 38, 0.16, False),
    (1, 28, 0.16, True),
    (3, 66, 0.16, False),   # a list long enough for several row tiles a warp
])
def test_residual_products(ccx, O, nmax, A, rho, snm):
    o = O.Oracle(O.Config(nmax=nmax, A=A, rho=rho, snm=snm, potential=int(snm)))
    e = ccx.Engine(ccx.Layout.from_basis(nmax, A, rho, snm=snm), real=not snm)
    e.generate(potential=ccx.POT_CHIRAL_LIKE if snm else ccx.POT_MINNESOTA)
    o.mp2()
    e.setup_t_amplitudes()
    o.t2_intermediate()
    e.t2_intermediate()
    n = o.n_channels(3)
    scale = max(np.abs(o.r2(c)).max(initial=0.0) for c in range(n))
    tol = 1e-11 if snm else 1e-12
    for c in range(n):
        assert np.abs(e.t2_eqn(c) - o.r2(c)).max(initial=0.0) < tol * scale, c
    for x, y in zip(e.denominators(), o.denoms()):
        assert np.abs(x - y).max() < tol * np.abs(y).max()
    o.close()
    e.close()
