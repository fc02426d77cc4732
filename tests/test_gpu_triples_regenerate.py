"""A second generated interaction reaches (T) as well: E(T) of a reused engine equals a fresh one's."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fp32", [True, False])
def test_triples_after_a_second_generation(ccx, fp32):
    L = ccx.Layout.from_basis(1, 4, 0.16, snm=True)

    def et(e, seed):
        e.generate(potential=ccx.POT_CHIRAL_LIKE, lec_seed=seed)
        e.setup_t_amplitudes()
        e.set_triples_precision(fp32=fp32)
        return e.pert_triples()

    a, b = ccx.Engine(L, real=False), ccx.Engine(L, real=False)
    first, second, want = et(a, 1), et(a, 2), et(b, 2)
    assert second == want and first != want
    a.close()
    b.close()
