"""The solver's products and guess block at the sizes where their launches change: the tall-skinny
product around its block counts, and solves whose guess block is a CSR block of the whole matrix
(97 rows and more) or the one-CTA Jacobi (fewer)."""
import numpy as np
import pytest

from helpers import gpu_context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 33, 4863, 4865, 38911, 38913, 160000])
@pytest.mark.parametrize("m,k", [(1, 1), (40, 8)])
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


@pytest.mark.parametrize("kw,ksym", [(dict(nbf=5, nelec=3), 1), (dict(nbf=6, nelec=4), 2), (dict(nbf=7, nelec=5), 1)])
@pytest.mark.parametrize("mixed", [False, True])
def test_roots_by_guess_block(kw, ksym, mixed):
    """60, 120 and 1,001 SEFs, against a dense eigen-solve of the stored matrix: residuals of 1e-8
    bound the roots' errors by 1e-8 squared over the gap, far below 1e-10."""
    import scipy.sparse as sp

    from psoci_gb300.inputs import make_problem

    c = gpu_context(make_problem("fci", seed=3, ksym=ksym, **kw))
    c.build_hamiltonian(mixed=mixed)
    rp, ci, va = c.get_hamiltonian()
    w = np.linalg.eigvalsh(sp.csr_matrix((va, ci, rp), shape=(c.nsef, c.nsef)).toarray())
    r = c.davidson(3, rtol=1e-8, mixed=mixed)
    assert np.abs(r.evals - w[:3]).max() <= 1e-10
    c.close()


@pytest.mark.parametrize("kw,nroots", [(dict(nbf=4, nelec=2), 1), (dict(nbf=5, nelec=3), 16), (dict(nbf=6, nelec=4), 9),
                                       (dict(nbf=7, nelec=5), 16), (dict(nbf=8, nelec=5), 8), (dict(nbf=9, nelec=5), 3)])
@pytest.mark.parametrize("max_subspace", [0, 48])
def test_orthonormal_vectors(kw, nroots, max_subspace):
    """Bases on both sides of 4,096 rows (one cluster's kernel below), 1 to 16 new vectors, with
    collapses (48 vectors): vectors orthonormal to the float-float sums (2^-45 of at most 1, well
    under 1e-12) and residuals as asked for."""
    import scipy.sparse as sp

    from psoci_gb300.inputs import make_problem

    c = gpu_context(make_problem("fci", seed=5, **kw))
    c.build_hamiltonian(mixed=False)
    rp, ci, va = c.get_hamiltonian()
    H = sp.csr_matrix((va, ci, rp), shape=(c.nsef, c.nsef))
    nroots = min(nroots, c.nsef)
    r = c.davidson(nroots, rtol=1e-8, mixed=False, max_subspace=max_subspace, want_vectors=True)
    v = r.evecs.reshape(nroots, c.nsef)
    assert np.abs(v @ v.T - np.eye(nroots)).max() <= 1e-12
    assert np.linalg.norm(H @ v.T - v.T * r.evals, axis=0).max() <= 2e-8
    c.close()
