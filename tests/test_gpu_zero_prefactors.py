"""Singles whose prefactor v0 is exactly zero while their exchange integrals are not: the reference
leaves the whole block out (PsociHamiltonian.C:239-258), and so do the build with listed pair
integrals, the one that evaluates them with the elements, and the direct product of either."""
import dataclasses

import numpy as np
import pytest

from helpers import check_h_against_oracle, gpu_context, small_problem

pytestmark = pytest.mark.gpu


def tri(a, b):
    return max(a, b) * (max(a, b) + 1) // 2 + min(a, b)


def exchange_only(p, rng):
    """(ip|pj) with i, p, j different, and orbital energies."""
    eri = np.zeros_like(p.eri)
    for i in range(p.nbf):
        for j in range(i):
            for q in range(p.nbf):
                if q not in (i, j):
                    eri[tri(tri(i, q), tri(q, j))] = rng.standard_normal()
    return dataclasses.replace(p, h=np.diag(rng.standard_normal(p.nbf)), eri=eri)


def small_integers(p, rng):
    """Integrals of -1, 0 and 1, so that sums cancel exactly, and orbital energies."""
    h = np.tril(rng.integers(-1, 2, p.h.shape), -1)
    return dataclasses.replace(p, h=h + h.T + np.diag(rng.standard_normal(p.nbf)), eri=rng.integers(-1, 2, p.eri.shape).astype(float))


@pytest.mark.parametrize("tables", [exchange_only, small_integers])
@pytest.mark.parametrize("name,ksym", [("fci_4e6o", 1), ("fci_5e6o", 2), ("fci_6e8o", 4)])
def test_zero_prefactor_is_skipped(oracle_mod, tables, name, ksym):
    p = tables(small_problem(name, ksym), np.random.default_rng(3))
    O = oracle_mod.Oracle(p)
    c = gpu_context(p)
    F = check_h_against_oracle(c, O, p, tol=1e-12)
    listed = c.get_hamiltonian()
    assert c.build_stats()["eval_launches"] == 2
    X = np.random.default_rng(9).standard_normal((c.nsef, 3))
    scale = abs(F).sum(axis=1).max() * np.abs(X).max()
    for launches in (0, 1):
        c.set_eval_launches(launches)
        c.build_hamiltonian(mixed=True)
        for a, b in zip(listed, c.get_hamiltonian()):
            assert np.array_equal(a, b)
        c.build_hamiltonian(direct=True)
        assert np.abs(c.sigma(X) - F @ X).max() <= 1e-14 * scale
    c.close()
