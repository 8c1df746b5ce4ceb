"""H from coupling tables at the edges of what the tables hold: 7 to 10 open shells (rows of
up to 256 SEFs, row offsets instead of 4-bit row counts), 11 open shells (the generic
kernels), doubly emptied and filled orbitals, two-word strings, both electron parities — the
stored matrix, and the direct product with no stored elements, against the oracle.

Elements are the reference's sums in its order, so they agree to rounding (a few ulps of
values up to about 50: 1e-12); products add at most a row of them."""
import numpy as np
import pytest

from helpers import check_h_against_oracle, gpu_context, lower_to_full, small_problem

pytestmark = pytest.mark.gpu


def neighbourhood(nbf, nelec, nopen, ksym, most, seed, shift=0):
    """A configuration with `nopen` open shells and its first `most` neighbours within two
    excitations (lexicographic order of the excitations), orbitals moved up by `shift`."""
    from psoci_gb300.inputs import Problem, config_jsym, make_integrals, make_irreps, select_block

    rng = np.random.default_rng(seed)
    n = nbf + shift
    irr = make_irreps(n, rng)
    h, so, eri = make_integrals(n, irr, n, rng)
    ref = np.zeros(n, np.uint8)
    ndbl = (nelec - nopen) // 2
    ref[shift:shift + ndbl] = 2
    ref[shift + ndbl:shift + ndbl + nopen] = 1
    occs = {tuple(ref)}
    singles = []
    for i in range(n):
        for a in range(n):
            o = ref.astype(int)
            o[i] -= 1
            o[a] += 1
            if i != a and o[i] >= 0 and o[a] <= 2:
                singles.append(tuple(o))
    rng.shuffle(singles)
    doubles = []
    for s in singles[:40]:
        for i, a in rng.integers(0, n, (6, 2)):
            o = np.array(s)
            o[i] -= 1
            o[a] += 1
            if i != a and o[i] >= 0 and o[a] <= 2:
                doubles.append(tuple(int(x) for x in o))
    for o in singles[:most // 2] + doubles:
        if len(occs) >= most:
            break
        if sum(x == 1 for x in o) <= 11:
            occs.add(tuple(int(x) for x in o))
    occ = np.array(sorted(occs, reverse=True), np.uint8)
    js = config_jsym(occ, irr)
    occ, js = select_block(occ, js, ksym)
    return Problem(nbf=n, nelec=nelec, ksym=ksym, mx_open=int((occ == 1).sum(1).max()), jsym=np.ascontiguousarray(js),
                   occ=np.ascontiguousarray(occ), h=h, so=so, eri=eri, irreps=irr)


CASES = {
    "open7": lambda: neighbourhood(9, 9, 7, 1, 60, 1),
    "open8": lambda: neighbourhood(10, 8, 8, 2, 40, 2),
    "open9": lambda: neighbourhood(11, 9, 9, 1, 16, 3),
    "open10": lambda: neighbourhood(11, 10, 10, 1, 10, 4),
    "open10_two_words": lambda: neighbourhood(11, 10, 8, 3, 24, 5, shift=58),
    "open11": lambda: neighbourhood(12, 11, 11, 2, 4, 6),
    "pairs": lambda: neighbourhood(8, 8, 0, 1, 120, 7),
    "one_electron": lambda: neighbourhood(6, 1, 1, 1, 6, 8),
    "two_electrons": lambda: small_problem("fci_4e6o", 2),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_tables_match_oracle(oracle_mod, name):
    p = CASES[name]()
    O = oracle_mod.Oracle(p)
    c = gpu_context(p)
    F = check_h_against_oracle(c, O, p, tol=1e-12)
    listed = c.get_hamiltonian()
    assert c.build_stats()["fast"] == (1 if p.mx_open <= 10 else 0)
    c.set_eval_launches(1)  # the pairs' integrals evaluated in the element launches
    c.build_hamiltonian(mixed=True)
    for a, b in zip(listed, c.get_hamiltonian()):
        assert np.array_equal(a, b)
    X = np.random.default_rng(9).standard_normal((c.nsef, 9))
    Y = F @ X
    c.build_hamiltonian(direct=True)
    scale = np.abs(F).sum(axis=1).max() * np.abs(X).max()
    assert np.abs(c.sigma(X) - Y).max() <= 1e-14 * scale
    c.close()


@pytest.mark.parametrize("name", ["open8", "open10", "open10_two_words", "open11", "pairs", "one_electron"])
@pytest.mark.parametrize("k", [1, 3, 9])
def test_gradient_contracts_to_the_energy(oracle_mod, name, k):
    """c^T H c is linear in the integrals, so the gradient contracted with them is the energy of
    each vector, with H from the oracle: 1, 3 and 9 vectors (a pass of eight and one of one); 11
    open shells go by the generic kernel.  Elements under the 1e-8 that H keeps are in the
    gradient and not in H: at most 1e-8 times |c|_1^2 <= 1e-8 N between the two."""
    p = CASES[name]()
    O = oracle_mod.Oracle(p)
    rp, ci, va = O.build_lower(4)
    v = np.random.default_rng(k).standard_normal((k, O.num_sefs()))
    v /= np.linalg.norm(v, axis=1)[:, None]
    F = lower_to_full(rp, ci, va, O.num_sefs())
    E = np.einsum("kn,kn->k", v, (F @ v.T).T)
    c = gpu_context(p)
    g1, g2 = c.energy_gradient(v)
    assert np.abs(g1 @ p.one_packed() + g2 @ p.eri - E).max() <= 1e-8 * O.num_sefs()
    c.close()


@pytest.mark.parametrize("k", [1, 9])
def test_gradient_matches_oracle(oracle_mod, k):
    """Doubly emptied and filled orbitals, entry by entry against the oracle's unit tables."""
    p = neighbourhood(5, 4, 0, 1, 12, 7)
    O = oracle_mod.Oracle(p)
    v = np.random.default_rng(k).standard_normal((k, O.num_sefs()))
    v /= np.linalg.norm(v, axis=1)[:, None]
    r1, r2 = O.energy_gradient(v)
    c = gpu_context(p)
    g1, g2 = c.energy_gradient(v)
    assert np.abs(g1 - r1).max() <= 1e-12 and np.abs(g2 - r2).max() <= 1e-12
    c.close()


@pytest.mark.parametrize("name", ["open8", "open10_two_words", "open11", "pairs", "one_electron"])
@pytest.mark.parametrize("k", [1, 2, 3, 9])
def test_density_matches_oracle(oracle_mod, name, k):
    """1-particle densities, passes of 1, 2, 4 and 8 roots; unit vectors, sums of at most N^2
    products of their entries."""
    p = CASES[name]()
    O = oracle_mod.Oracle(p)
    v = np.random.default_rng(k).standard_normal((k, O.num_sefs()))
    v /= np.linalg.norm(v, axis=1)[:, None]
    c = gpu_context(p)
    assert np.abs(c.density1(v) - O.density1(v)).max() <= 1e-12
    c.close()


@pytest.mark.parametrize("nbf,nelec,nopen", [(3, 4, 0), (4, 5, 1), (4, 6, 2), (5, 5, 3), (66, 6, 4), (6, 6, 6), (9, 9, 7)])
@pytest.mark.parametrize("ksym", [1, 2])
@pytest.mark.parametrize("prec", [0, 1])
def test_gradient_of_one_configuration(oracle_mod, nbf, nelec, nopen, ksym, prec):
    """A diagonal block alone, in either symmetry block (the second determinants' sign), by the
    closed form of its derivatives: E = sum occ h_ii + (ii|ii) of doubly occupied + pairs, the
    exchange of two open shells from the oracle's element with that integral alone.  Unit vectors;
    FP32 sums of at most 2^6 squares and products err by less than 2^6 2^-24 times their norm."""
    p = neighbourhood(8 if nbf == 66 else nbf, nelec, nopen, 1, 1, 3, shift=58 if nbf == 66 else 0)
    p.ksym = ksym
    O = oracle_mod.Oracle(p)
    N = O.num_sefs()
    v = np.random.default_rng(nopen).standard_normal((3, N))
    v /= np.linalg.norm(v, axis=1)[:, None]
    c = gpu_context(p)
    g1, g2 = c.energy_gradient(v, prec=prec)
    c.close()
    occ = p.occ[0].astype(int)
    tri = lambda a, b: max(a, b) * (max(a, b) + 1) // 2 + min(a, b)
    r1, r2 = np.zeros_like(g1), np.zeros_like(g2)
    orb = np.flatnonzero(occ)
    for i in orb:
        r1[:, tri(i, i)] += occ[i]
        if occ[i] == 2:
            r2[:, tri(tri(i, i), tri(i, i))] += 1.0
        for j in orb[orb < i]:
            r2[:, tri(tri(i, i), tri(j, j))] += occ[i] * occ[j]
            if occ[i] * occ[j] > 1:
                r2[:, tri(tri(i, j), tri(i, j))] -= occ[i] * occ[j] / 2
            else:
                q = oracle_mod.Oracle(_only(p, tri(tri(i, j), tri(i, j))))
                F = lower_to_full(*q.build_lower(1), N)
                r2[:, tri(tri(i, j), tri(i, j))] += np.einsum("kn,kn->k", v, (F @ v.T).T)
    tol = 2.0 ** -18 if prec else 1e-13
    assert np.abs(g1 - r1).max() <= tol * 2 and np.abs(g2 - r2).max() <= tol * 4


def _only(p, at):
    """p with one two-electron integral, 1, and nothing else."""
    import dataclasses

    eri = np.zeros_like(p.eri)
    eri[at] = 1.0
    return dataclasses.replace(p, h=np.zeros_like(p.h), so=np.zeros_like(p.so), eri=eri)
