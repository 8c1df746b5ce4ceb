"""Calls within a limit on the context's device memory.  What the coupling tables and pair lists take is
not needed: where it does not fit, the calls go by the kernels that need neither, to the same
results, and what a call keeps for its speed is given back to one that needs the room."""
import numpy as np
import pytest

from helpers import gpu_context, small_problem

pytestmark = pytest.mark.gpu


def unit_vectors(k, n):
    v = np.random.default_rng(k).standard_normal((k, n))
    return v / np.linalg.norm(v, axis=1)[:, None]


def least_room(p, call, check):
    """Bytes beyond a fresh context's from which on call(c) runs, in steps of a quarter, then to 2%; its
    results are checked at each step.  And the bytes that it leaves in use without a limit."""
    from psoci_gb300 import api

    c = gpu_context(p)
    held = c.set_memory_limit(0)
    check(call(c))
    kept = c.set_memory_limit(0) - held
    c.close()

    def runs(room):
        c = gpu_context(p)
        c.set_memory_limit(c.set_memory_limit(0) + room)
        try:
            r = call(c)
        except api.PsociError as e:
            assert "memory" in str(e), e
            return False
        else:
            check(r)
            return True
        finally:
            c.close()

    rooms = [int((1 << 15) * 1.25 ** q) for q in range(34)]  # to 52 MB
    ok = [runs(r) for r in rooms]
    first = ok.index(True)
    assert all(ok[first:])
    lo, hi = rooms[first] * 4 // 5, rooms[first]
    while hi - lo > hi // 50:
        mid = (lo + hi) // 2
        lo, hi = (lo, mid) if runs(mid) else (mid, hi)
    return hi, kept


def test_limit_is_kept():
    """A build that cannot fit is refused, and runs again once the limit is gone."""
    from psoci_gb300 import api

    c = gpu_context(small_problem("fci_6e8o", 1))
    c.set_memory_limit(c.set_memory_limit(0) + (1 << 20))
    with pytest.raises(api.PsociError, match="memory"):
        c.build_hamiltonian(mixed=True)
    c.set_memory_limit(0)
    assert c.build_hamiltonian(mixed=True) > 0
    c.close()


@pytest.mark.parametrize("k", [1, 5])
@pytest.mark.parametrize("name,ksym", [("fci_5e6o", 1), ("fci_6e8o", 1)])
def test_density(oracle_mod, name, ksym, k):
    """Runs in less than what its plan and rows take where there is room."""
    p = small_problem(name, ksym)
    O = oracle_mod.Oracle(p)
    v = unit_vectors(k, O.num_sefs())
    ref = O.density1(v)
    rows = 2 * v.nbytes  # the vectors of the call, kept
    least, kept = least_room(p, lambda c: c.density1(v), lambda d: np.testing.assert_allclose(d, ref, rtol=0, atol=1e-12))
    assert least - rows < 0.8 * (kept - rows)


@pytest.mark.parametrize("k", [1, 5])
@pytest.mark.parametrize("nonzero", [False, True])
def test_gradient(k, nonzero):
    """Sums of at most N^2 products of unit vectors in either kernel; runs in less than what the lists
    and tables take."""
    p = small_problem("fci_6e8o", 1)
    c = gpu_context(p)
    v = unit_vectors(k, c.nsef)
    ref = c.energy_gradient(v, nonzero_only=nonzero)
    c.close()

    def check(g):
        for a, b in zip(ref, g):
            assert np.abs(a - b).max() <= 1e-12

    least, kept = least_room(p, lambda c: c.energy_gradient(v, nonzero_only=nonzero), check)
    assert least < kept + (1 << 17)  # the call's vectors and screen beside them


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
    """From no room for the tables to room for everything: the matrix without a limit to rounding (the
    generic kernels form an element's sum in the reference's order, as the tables do), and the direct
    product.  The generic build needs the matrix and little else; the direct build less than what it
    keeps where there is room."""
    p = small_problem(name, ksym)
    c = gpu_context(p)
    nnz = c.build_hamiltonian(mixed=True)
    m = c.get_hamiltonian()
    x = unit_vectors(3, c.nsef).T.copy()
    y = c.sigma(x)
    scale = np.abs(m[2]).max() * np.diff(m[0]).max()
    c.close()
    forms = set()

    def stored(c):
        c.build_hamiltonian(mixed=True)
        st = c.build_stats()
        forms.add(st["eval_launches"])
        assert st["fast"] == (st["eval_launches"] > 0)
        return c.get_hamiltonian()

    def same(g):
        assert np.array_equal(m[0], g[0]) and np.array_equal(m[1], g[1])
        assert np.abs(m[2] - g[2]).max() <= 1e-12

    least_room(p, stored, same)
    assert {0, 2} <= forms

    def direct(c):
        c.build_hamiltonian(direct=True)
        return c.sigma(x)

    def close(z):
        assert np.abs(y - z).max() <= 1e-14 * scale

    least, kept = least_room(p, direct, close)
    assert least < kept
    assert nnz == m[0][-1]


@pytest.mark.parametrize("mixed", [False, True])
def test_direct_solve_takes_the_tables_memory(mixed):
    """A direct build's pair integrals, then its tables, go when the solve's basis needs their room: the
    solve runs beside all, 60% and 30% of what the build holds (its lists, which stay, are 10%)."""
    p = small_problem("fci_6e8o", 1)
    c = gpu_context(p)
    c.build_hamiltonian(direct=True)
    full = c.davidson(4, rtol=1e-8, mixed=mixed, max_subspace=12).evals
    c.close()
    left = []
    for share in (1.0, 0.6, 0.3):
        c = gpu_context(p)
        before = c.set_memory_limit(0)
        c.build_hamiltonian(direct=True)
        held = c.set_memory_limit(0)
        basis = c.nsef * 8 * (2 * 12 + 6 * 4 + 2 * 4) + (1 << 19)  # V, HV; X, R, T, tmp; staging; sums
        c.set_memory_limit(before + int(share * (held - before)) + basis)
        r = c.davidson(4, rtol=1e-8, mixed=mixed, max_subspace=12)
        assert np.abs(r.evals - full).max() <= 1e-10
        left.append(held - c.set_memory_limit(0))
        c.close()
    assert left[0] < left[1] <= left[2]


def test_build_takes_the_densitys_memory():
    p = small_problem("fci_6e8o", 1)
    least, _ = least_room(p, lambda c: c.build_hamiltonian(mixed=True), lambda n: None)
    c = gpu_context(p)
    v = unit_vectors(2, c.nsef)
    before = c.set_memory_limit(0)
    d = c.density1(v)
    held = c.set_memory_limit(0)
    c.set_memory_limit(held + least - (held - before - 2 * v.nbytes) // 2)
    c.build_hamiltonian(mixed=True)
    c.set_memory_limit(0)
    assert np.abs(c.density1(v) - d).max() <= 1e-14
    c.close()
