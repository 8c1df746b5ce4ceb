"""The FP32 and float-float products at every width of the vector block: each has its own row of the
staged inputs (1, 2, 4 or 8 entries) and block size, and 9 is a full chunk and a ragged one."""
import numpy as np
import pytest

from helpers import gpu_context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [dict(nbf=5, nelec=3), dict(nbf=7, nelec=5)])
def test_products_by_width(kw):
    """Against FP64 products of the stored matrix, element by element.  With m elements a lane: the
    mixed product rounds element, input and product to FP32 (3 units of 2^-24) and its compensated sums
    add two more; float-float keeps 48 bits of each factor, drops the low x low product and adds its low
    words in FP32 (at most m units of 2^-47)."""
    import scipy.sparse as sp

    from psoci_gb300.inputs import make_problem

    c = gpu_context(make_problem("fci", seed=3, **kw))
    c.build_hamiltonian(mixed=True)
    rp, ci, va = c.get_hamiltonian()
    H = sp.csr_matrix((va, ci, rp), shape=(c.nsef, c.nsef))
    m = -(-int(np.diff(rp).max()) // 32)
    rng = np.random.default_rng(5)
    for k in range(1, 10):
        X = rng.standard_normal((c.nsef, k))
        ref, scale = H @ X, abs(H) @ np.abs(X)
        assert (np.abs(c.sigma(X, prec=1) - ref) <= 6 * 2.0 ** -24 * scale).all()
        assert (np.abs(c.sigma(X, prec=2) - ref) <= (m + 6) * 2.0 ** -47 * scale).all()
    c.close()
