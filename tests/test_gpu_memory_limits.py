"""Calls within a limit on the context's device memory: what the coupling tables and pair lists would
take is not there (3 MB beyond what the call's inputs hold; the tables alone start at 4 MB), so the
calls go by the kernels that need neither, to the same results."""
import numpy as np
import pytest

from helpers import gpu_context, small_problem

pytestmark = pytest.mark.gpu

ROOM = 3 << 20


def unit_vectors(k, n):
    v = np.random.default_rng(k).standard_normal((k, n))
    return v / np.linalg.norm(v, axis=1)[:, None]


def limited(p, room=ROOM):
    c = gpu_context(p)
    held = c.set_memory_limit(0)
    c.set_memory_limit(held + room)
    return c


def test_limit_is_kept():
    """A build that cannot fit is refused, and runs again once the limit is gone."""
    from psoci_gb300 import api

    c = limited(small_problem("fci_6e8o", 1), 1 << 20)
    with pytest.raises(api.PsociError, match="memory"):
        c.build_hamiltonian(mixed=True)
    c.set_memory_limit(0)
    assert c.build_hamiltonian(mixed=True) > 0
    c.close()


@pytest.mark.parametrize("k", [1, 5])
@pytest.mark.parametrize("name,ksym", [("fci_5e6o", 1), ("fci_6e8o", 1)])
def test_density(oracle_mod, name, ksym, k):
    p = small_problem(name, ksym)
    O = oracle_mod.Oracle(p)
    v = unit_vectors(k, O.num_sefs())
    c = limited(p)
    assert np.abs(c.density1(v) - O.density1(v)).max() <= 1e-12
    c.close()
