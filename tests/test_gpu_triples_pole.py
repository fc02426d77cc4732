"""A vanishing denominator in (T): one infinite term makes the sum infinite, not a NaN, with either
contractions."""
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_one_vanishing_denominator(ccx):
    L = ccx.Layout.from_basis(1, 3, 0.08, theta=(0.7, 0.2, -0.4))  # one hole triple
    orb = L.orbits()
    n = np.stack([orb[k] for k in ("nx", "ny", "nz")], axis=1)
    e = ccx.Engine(L, real=True)
    e.generate()
    e.setup_t_amplitudes()
    ns, rng = len(n), np.random.RandomState(3)
    total, found = n[:3].sum(0), 0
    for t in itertools.combinations(range(3, ns), 3):
        if np.any(n[list(t)].sum(0) != total):
            continue
        f = np.concatenate([[-3.0, -5.0, -7.0], rng.uniform(50.0, 90.0, ns - 3)])
        f[list(t)] = (-2.0, -6.0, -7.0)  # the same sum as the holes'
        e.set_fock(np.diag(f).astype(complex))
        e.set_triples_precision(fp32=False)
        if not np.isinf(e.pert_triples().real):  # this triple has no amplitude
            continue
        e.set_triples_precision(fp32=True)
        assert np.isinf(e.pert_triples().real), t
        found += 1
        if found == 3:
            break
    assert found
    e.close()
