"""The solver's launches where they change: the tall-skinny product at 76 and 608 blocks of 256 rows
(two and eight outputs a thread, blocks of more rows), and the orthonormalisation at 4,096 rows
(one cluster's kernel below)."""
import ctypes

import numpy as np
import pytest

from helpers import gpu_context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [255, 256, 257, 19455, 19456, 19457, 155647, 155648, 155649])
@pytest.mark.parametrize("m,k", [(40, 8), (3, 7), (40, 5)])
def test_tall_skinny_product(n, m, k):
    """C = A^T B in float-float: products and sums good to about 2^-45 of sum |a||b|."""
    torch = pytest.importorskip("torch")
    from psoci_gb300 import api

    rng = np.random.default_rng(n)
    A, B = rng.standard_normal((n, m)), rng.standard_normal((n, k))
    dA, dB = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    dC = torch.empty((m, k), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    with api.Context(0) as c:
        c.tsprod_device(0, n, dA.data_ptr(), m, m, dB.data_ptr(), k, k, dC.data_ptr())
    scale = np.abs(A).T @ np.abs(B)
    assert (np.abs(dC.cpu().numpy() - A.T @ B) <= 2.0 ** -44 * scale).all()


def problem_of_rows(rows):
    """Configurations of 5 electrons in 9 orbitals, as many as make `rows` SEFs."""
    import dataclasses

    from psoci_gb300.inputs import make_problem

    p = make_problem("fci", nbf=9, nelec=5, seed=5)
    nsef = 2 ** (p.nopen() - 1)
    take = np.cumsum(nsef) <= rows - 100
    left = rows - nsef[take].sum()
    for i in np.flatnonzero(~take):
        if nsef[i] <= left:
            take[i] = True
            left -= nsef[i]
    assert left == 0
    return dataclasses.replace(p, occ=np.ascontiguousarray(p.occ[take]), jsym=np.ascontiguousarray(p.jsym[take]))


@pytest.mark.parametrize("rows", [4095, 4096, 4097])
@pytest.mark.parametrize("k", [1, 8, 16])
def test_orthonormal_set(rows, k):
    """A set of random vectors: orthonormal to float-float sums (well under 1e-12), of the same span."""
    c = gpu_context(problem_of_rows(rows))
    c.build_hamiltonian(mixed=False)
    assert c.nsef == rows
    v = np.random.default_rng(k).standard_normal((k, rows))
    c.set_guess(v)
    lib = c.lib
    assert lib.psoci_basis_create(c.ctx, k, k + 1) == 0
    assert lib.psoci_basis_guess(c.ctx, 2) == 0
    assert lib.psoci_basis_orthonormalize_all(c.ctx, None) == 0
    q = np.zeros((k, rows))
    assert lib.psoci_basis_vectors(c.ctx, k, q.ctypes.data_as(ctypes.POINTER(ctypes.c_double))) == 0
    c.close()
    assert np.abs(q @ q.T - np.eye(k)).max() <= 1e-12
    assert np.abs(v - (v @ q.T) @ q).max() <= 1e-11


@pytest.mark.parametrize("nbf,nroots", [(2, 3), (3, 6), (5, 15), (6, 16)])
@pytest.mark.parametrize("mixed", [False, True])
def test_many_roots_of_few_rows(nbf, nroots, mixed):
    """All of 3, 6 and 15 roots and 16 of 21, against a dense eigen-solve: residuals of 1e-8."""
    import scipy.sparse as sp

    from psoci_gb300.inputs import make_problem

    c = gpu_context(make_problem("fci", nbf=nbf, nelec=2, seed=3))
    c.build_hamiltonian(mixed=mixed)
    rp, ci, va = c.get_hamiltonian()
    w = np.linalg.eigvalsh(sp.csr_matrix((va, ci, rp), shape=(c.nsef, c.nsef)).toarray())
    r = c.davidson(nroots, rtol=1e-8, mixed=mixed)
    assert np.abs(r.evals - w[:nroots]).max() <= 1e-8
    c.close()
