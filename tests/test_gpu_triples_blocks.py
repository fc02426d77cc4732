"""(T) over momentum blocks against the oracle: both numbers of isospins, real and complex, shells
that are partly filled (a momentum with hole and particle states), lattices with few blocks.

FP64 contractions in another order than the oracle's: 1e-10 of E(T), as the other comparisons.  FP32
contractions: 1e-5 (the accuracy asked of them)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nmax,A,snm,pot,real,theta", [
    (1, 14, False, 0, True, (0.0, 0.0, 0.0)),
    (1, 7, False, 0, True, (0.0, 0.0, 0.0)),     # a hole and a particle state on one momentum
    (1, 3, False, 0, True, (0.7, 0.2, -0.4)),    # one hole triple
    (1, 2, False, 0, True, (0.0, 0.0, 0.0)),     # none
    (2, 14, False, 0, False, (0.3, -1.0, 0.6)),  # one isospin in a complex engine
    (1, 6, True, 0, True, (0.0, 0.0, 0.0)),      # two isospins, real, partly filled
    (1, 4, True, 1, False, (0.0, 0.0, 0.0)),
    (1, 28, True, 1, False, (0.5, -0.3, 1.2)),
])
def test_triples_blocks(ccx, O, nmax, A, snm, pot, real, theta):
    rho = 0.08 if not snm else 0.16
    o = O.Oracle(O.Config(nmax=nmax, A=A, rho=rho, snm=snm, theta=theta, potential=pot))
    e = ccx.Engine(ccx.Layout.from_basis(nmax, A, rho, snm=snm, theta=theta), real=real)
    e.generate(potential=pot)
    o.mp2()
    e.setup_t_amplitudes()
    want = o.triples()
    got32 = e.pert_triples()
    e.set_triples_precision(fp32=False)
    got = e.pert_triples()
    assert abs(got - want) <= 1e-10 * abs(want), (got, want)
    assert abs(got32 - want) <= 1e-5 * abs(want), (got32, want)
    o.close()
    e.close()


def test_triples_of_fresh_engines_repeat(ccx):
    """Every engine's first (T) is the same: its tables and zeroed buffers are in place before its
    kernels run (each engine sets them up on another stream than it computes on)."""
    L = ccx.Layout.from_basis(2, 4, 0.16, snm=True)
    got = set()
    for fp32 in [True, False] * 10:
        e = ccx.Engine(L, real=False)
        e.generate(potential=ccx.POT_CHIRAL_LIKE)
        e.setup_t_amplitudes()
        e.set_triples_precision(fp32=fp32)
        got.add((fp32, e.pert_triples()))
        e.close()
    assert len(got) == 2, got
