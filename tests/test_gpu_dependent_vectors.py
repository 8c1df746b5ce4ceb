"""Orthonormalisation of guess sets with dependent vectors: of 9 to 16 vectors 1 to 12 are
independent, the others are dropped, and the second pass runs on fewer columns than the set
came with.  The independent vectors have disjoint supports of 4 or 64 rows and entries of +-1,
the dependent ones are copies, negatives and zeros, so every sum and pivot is exact: dependent
pivots are exactly zero, and the kept vectors are the inputs over 2 or 8 to the bit."""
import ctypes

import numpy as np
import pytest

from helpers import gpu_context

pytestmark = pytest.mark.gpu

PSOCI_ERR_NUMERIC = 8


@pytest.mark.parametrize("kw,support", [(dict(nbf=6, nelec=4), 4), (dict(nbf=7, nelec=5), 64), (dict(nbf=8, nelec=5), 64)])
@pytest.mark.parametrize("b,rank", [(9, 1), (9, 8), (12, 4), (13, 8), (16, 1), (16, 4), (16, 8), (16, 12)])
def test_dependent_vectors_are_dropped(kw, support, b, rank):
    from psoci_gb300.inputs import make_problem

    c = gpu_context(make_problem("fci", seed=5, ksym=2, **kw))
    c.build_hamiltonian(mixed=False)
    N = c.nsef
    rng = np.random.default_rng(16 * b + rank)
    rows = rng.permutation(N)[: rank * support].reshape(rank, support)
    ind = np.zeros((rank, N))
    for j in range(rank):
        ind[j, rows[j]] = rng.choice([-1.0, 1.0], support)
    # the independent ones in order, copies of earlier ones (or zeros) in between
    place = np.sort(np.concatenate([[0], 1 + rng.permutation(b - 1)[: rank - 1]]))
    v = np.zeros((b, N))
    v[place] = ind
    for j in set(range(b)) - set(place.tolist()):
        v[j] = ind[rng.integers(np.count_nonzero(place < j))] * rng.choice([-1.0, 0.0, 1.0])
    c.set_guess(v)
    lib, at = c.lib, ctypes.c_int()
    assert lib.psoci_basis_create(c.ctx, b, b + 1) == 0
    assert lib.psoci_basis_guess(c.ctx, 2) == 0
    assert lib.psoci_basis_orthonormalize_all(c.ctx, ctypes.byref(at)) == PSOCI_ERR_NUMERIC
    assert at.value == rank + 1
    out = np.zeros((rank, N))
    assert lib.psoci_basis_vectors(c.ctx, rank, out.ctypes.data_as(ctypes.POINTER(ctypes.c_double))) == 0
    assert np.array_equal(out, ind / np.sqrt(support))
    c.close()


@pytest.mark.parametrize("kw", [dict(nbf=6, nelec=4), dict(nbf=9, nelec=5)])
@pytest.mark.parametrize("nroots,copies", [(3, 3), (9, 9), (16, 12)])
@pytest.mark.parametrize("mixed", [False, True])
def test_restart_from_copies(kw, nroots, copies, mixed):
    """Restart vectors that are copies of one: the roots are those of a solve without them."""
    from psoci_gb300.inputs import make_problem

    c = gpu_context(make_problem("fci", seed=5, ksym=2, **kw))
    c.build_hamiltonian(mixed=mixed)
    free = c.davidson(nroots, rtol=1e-8, mixed=mixed)
    v = np.zeros((copies, c.nsef))
    v[:, 7] = 1.0
    c.set_guess(v)
    r = c.davidson(nroots, rtol=1e-8, mixed=mixed)
    assert np.abs(r.evals - free.evals).max() <= 1e-9
    c.close()
