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


@pytest.mark.parametrize("k", [1, 5])
@pytest.mark.parametrize("room", [ROOM, 1 << 20])
@pytest.mark.parametrize("nonzero", [False, True])
def test_gradient(room, k, nonzero):
    """Sums of at most N^2 products of unit vectors in either kernel."""
    p = small_problem("fci_5e6o", 1)
    c = gpu_context(p)
    v = unit_vectors(k, c.nsef)
    free = c.energy_gradient(v, nonzero_only=nonzero)
    c.close()
    c = limited(p, room)
    for a, b in zip(free, c.energy_gradient(v, nonzero_only=nonzero)):
        assert np.abs(a - b).max() <= 1e-12
    c.close()


def test_gradient_vectors_without_room():
    """The lists, tables and eight vectors with their gradients (172 KB) have room, the vectors' rows
    (128 KB) beside them do not."""
    p = small_problem("fci_6e8o", 1)
    c = gpu_context(p)
    v = unit_vectors(8, c.nsef)
    free = c.energy_gradient(v)
    c.close()
    c = gpu_context(p)
    c.energy_gradient(v[:1])  # the plan, and a first pass
    c.set_memory_limit(c.set_memory_limit(0) + (240 << 10))
    for a, b in zip(free, c.energy_gradient(v)):
        assert np.abs(a - b).max() <= 1e-12
    c.close()


@pytest.mark.parametrize("name,ksym", [("fci_5e6o", 1), ("fci_6e8o", 1)])
def test_build_and_direct_product(name, ksym):
    """From room for everything to none for the tables: the matrix without a limit to rounding (the
    generic kernels form an element's sum in the reference's order, as the tables do), and the direct
    product."""
    p = small_problem(name, ksym)
    c = gpu_context(p)
    nnz = c.build_hamiltonian(mixed=True)
    rp, ci, va = c.get_hamiltonian()
    x = unit_vectors(3, c.nsef).T.copy()
    y = c.sigma(x)
    scale = np.abs(va).max() * np.diff(rp).max()
    c.close()
    stored = set()
    for room in [64 << 20] + [(ROOM + 16 * nnz) + (q << 19) for q in range(16)]:
        c = limited(p, room)
        c.build_hamiltonian(mixed=True)
        st = c.build_stats()
        stored.add(st["eval_launches"])
        assert st["fast"] == (st["eval_launches"] > 0)
        for a, b in zip((rp, ci), c.get_hamiltonian()):
            assert np.array_equal(a, b)
        assert np.abs(c.get_hamiltonian()[2] - va).max() <= 1e-12
        c.build_hamiltonian(direct=True)
        assert np.abs(c.sigma(x) - y).max() <= 1e-14 * scale
        c.close()
    assert {0, 2} <= stored
    c = limited(p, ROOM)
    c.build_hamiltonian(direct=True)
    assert np.abs(c.sigma(x) - y).max() <= 1e-14 * scale
    c.close()


@pytest.mark.parametrize("below", [-(1 << 18), 0, 3 << 20])
@pytest.mark.parametrize("mixed", [False, True])
def test_direct_solve_takes_the_tables_memory(below, mixed):
    """A direct build's pair integrals, then its tables, go when the solve's basis (2 MB) needs their
    room: limits of 256 KB above to 3 MB below what the build holds."""
    p = small_problem("fci_6e8o", 1)
    c = gpu_context(p)
    c.build_hamiltonian(direct=True)
    full = c.davidson(4, rtol=1e-8, mixed=mixed)
    c.close()
    c = gpu_context(p)
    c.build_hamiltonian(direct=True)
    held = c.set_memory_limit(0)
    c.set_memory_limit(held - below)
    r = c.davidson(4, rtol=1e-8, mixed=mixed)
    assert np.abs(r.evals - full.evals).max() <= 1e-10
    assert c.set_memory_limit(0) < held - max(below, 0)
    c.close()


def test_build_takes_the_densitys_memory():
    p = small_problem("fci_6e8o", 1)
    c = gpu_context(p)
    v = unit_vectors(2, c.nsef)
    d = c.density1(v)
    c.set_memory_limit(c.set_memory_limit(0) + (1 << 20))
    c.build_hamiltonian(mixed=True)  # 3.4 MB of elements
    c.set_memory_limit(0)
    assert np.abs(c.density1(v) - d).max() <= 1e-14
    c.close()
