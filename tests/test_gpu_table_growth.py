"""Coupling tables beyond the words that a first build starts with (2^20): the tables are made again
in a larger pool, with the pairs' slots of the first attempt, and each of the build, the density and
the gradient remembers its own size."""
import numpy as np
import pytest

from helpers import gpu_context
from test_gpu_coupling_tables import neighbourhood

pytestmark = pytest.mark.gpu


def test_pool_grows_once():
    p = neighbourhood(13, 10, 10, 1, 250, 4)
    c = gpu_context(p)
    lib = c.lib

    def build():
        n = lib.psoci_launch_count()
        c.build_hamiltonian(mixed=True)
        return lib.psoci_launch_count() - n

    first = build()  # one table launch more: the pool of 2^20 words is too small
    m = c.get_hamiltonian()
    assert build() == first - 1
    for a, b in zip(m, c.get_hamiltonian()):
        assert np.array_equal(a, b)
    v = np.random.default_rng(1).standard_normal((2, c.nsef))
    v /= np.linalg.norm(v, axis=1)[:, None]
    d = c.density1(v)  # fewer words than the build
    assert build() == first - 1
    assert np.array_equal(m[2], c.get_hamiltonian()[2])
    # trace of a density: the electrons
    tri = np.cumsum(np.arange(1, p.nbf + 1)) - 1
    assert np.abs(d[:, tri].sum(axis=1) - p.nelec).max() <= 1e-12
    c.close()
