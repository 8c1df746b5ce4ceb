"""Energy gradients of one, two, four and eight roots a pass, and of a pass and a rest: of all integrals
and of the non-zero ones alone, which are the same where the integral is not zero, and zero where
it is.  Sums of at most N^2 products of unit vectors' entries, in another order: 1e-12."""
import numpy as np
import pytest

from helpers import gpu_context, small_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,ksym", [("fci_5e6o", 2), ("fci_6e8o", 1)])
def test_passes_of_roots(name, ksym):
    p = small_problem(name, ksym)
    c = gpu_context(p)
    v = np.random.default_rng(2).standard_normal((9, c.nsef))
    v /= np.linalg.norm(v, axis=1)[:, None]
    each = [c.energy_gradient(x[None]) for x in v]
    tabs = (p.one_packed(), p.eri)
    for k in (1, 2, 3, 4, 8, 9):
        for nonzero in (False, True):
            for i, g in enumerate(c.energy_gradient(v[:k], nonzero_only=nonzero)):
                ref = np.concatenate([e[i] for e in each[:k]])
                if nonzero:
                    ref = np.where(tabs[i] != 0, ref, 0.0)
                    assert not g[:, tabs[i] == 0].any()
                assert np.abs(g - ref).max() <= 1e-12
    c.close()
