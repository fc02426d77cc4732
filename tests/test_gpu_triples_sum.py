"""(T) with FP32 contractions: the sum over the pairs keeps FP64's accuracy, however many."""
import pytest

pytestmark = pytest.mark.gpu


def test_fp32_contractions_sum(ccx):
    """Rounded terms (6e-8 each, of both signs) average out over 3e10 pairs; what is left is their
    bias, 7.3e-10 where every term is added in FP64.  Terms lost from the sum are all of one sign
    and add up: below 3e-9 of E(T)."""
    e = ccx.Engine(ccx.Layout.from_basis(3, 132, 0.16, snm=True), real=False)
    e.generate(potential=ccx.POT_CHIRAL_LIKE)
    e.setup_t_amplitudes()
    got32 = e.pert_triples()
    e.set_triples_precision(fp32=False)
    got64 = e.pert_triples()
    e.close()
    assert abs(got32 - got64) < 3e-9 * abs(got64)
