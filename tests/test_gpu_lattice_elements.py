"""Interaction generated from the lattice tables against the element-by-element form.

An orbital moved off the momentum lattice by 1e-12 of its momentum makes the engine evaluate
every element in full; the elements then differ by that shift (times at most q^2 / kappa < 100
for the steepest Gaussian) and by rounding, so blocks agree to 1e-10 of their largest entry.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nmax,A,snm,pot,real,theta", [
    (1, 2, False, 0, True, (0.0, 0.0, 0.0)),      # one pair tile
    (2, 14, False, 0, True, (0.3, -1.1, 2.0)),    # ragged 32 x 32 tiles, twisted
    (1, 4, True, 0, False, (0.0, 0.0, 0.0)),      # Minnesota in a complex engine, both isospins
    (1, 28, True, 1, False, (0.5, 0.1, -2.5)),
    (2, 4, True, 1, False, (0.0, 0.0, 0.0)),
])
def test_lattice_tables_match_elements_in_full(ccx, nmax, A, snm, pot, real, theta):
    L = ccx.Layout.from_basis(nmax, A, 0.16, snm=snm, theta=theta)
    orb = L.orbits()
    moved = {k: np.array(v) for k, v in orb.items() if k not in ("n_holes", "box_length")}
    moved["kx"][-1] *= 1.0 + 1e-12
    L2 = ccx.Layout.from_orbits(moved, A, orb["box_length"])
    engines = []
    for lay in (L, L2):
        e = ccx.Engine(lay, real=real)
        e.generate(potential=pot)
        e.setup_t_amplitudes()
        e.t2_intermediate()
        engines.append(e)
    a, b = engines

    def close(x, y, what):
        x, y = np.asarray(x), np.asarray(y)
        assert np.abs(x - y).max(initial=0.0) <= 1e-10 * max(np.abs(y).max(initial=0.0), 1e-6), what

    close(a.e0(), b.e0(), "e0")
    close(a.fock(), b.fock(), "fock")
    close(a.ccd_energy(), b.ccd_energy(), "mp2")
    c = L.counts()
    for kind, n in ((ccx.CH_HHPP, c["hhpp"]), (ccx.V_PPPP, c["hhpp"]), (ccx.CH_HHHH, c["hhhh"]),
                    (ccx.CH_HPHP, c["hphp"])):
        for ch in range(0, n, max(1, n // 8)):
            close(a.vblock(kind, ch), b.vblock(kind, ch), (kind, ch))
    # the stored blocks, through every product of the residual
    scale = max(np.abs(b.t2_eqn(ch)).max(initial=0.0) for ch in range(c["hhpp"]))
    for ch in range(c["hhpp"]):
        assert np.abs(a.t2_eqn(ch) - b.t2_eqn(ch)).max(initial=0.0) <= 1e-9 * scale, ch
    close(a.pert_triples(), b.pert_triples(), "triples")
