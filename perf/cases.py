"""The work that a user of this package has it do, as cases that can be timed and compared.

A program sets one symmetry block's integrals and configurations, builds its determinants
and Hamiltonian, takes H-times-vector products or whole eigen-solves from it, and forms
densities and energy gradients from the vectors.  Each case is one of these calls through
``psoci_gb300.api``:

  sigma     Y = H X from the stored matrix, device pointers (a host's own eigensolver loop)
  direct    the same product without a stored matrix
  build     determinants and stored Hamiltonian, then the first product with it
  solve     new inputs to eigenvalues: integrals, configurations, determinants, H, Davidson
  density   1-particle densities of CI vectors
  gradient  1- and 2-particle densities (dE / d integrals) of CI vectors

Spaces are the families of ``psoci_gb300.inputs`` (full CI, and a full-CI reference plus
singles or singles and doubles into virtuals) with its seeded integrals.
"""
import math

import numpy as np
import torch

from psoci_gb300 import api
from psoci_gb300.inputs import make_problem

PREC = {"fp64": api.PREC_FP64, "mixed": api.PREC_MIXED, "ff": api.PREC_FF}


def _space(kind, nact, nelec, nvirt=0, ksym=1):
    return {"space": kind, "nact": nact, "nelec": nelec, "nvirt": nvirt, "ksym": ksym}


def listed():
    return [
        # 4 vectors of a small full-CI block: the smallest call, where latency counts
        dict(name="sigma_fci_k4", do="sigma", prec="fp64", k=4, **_space("fci", 8, 6)),
        # the 8-root block of a singles CI in FP32 elements: the ordinary call of a mixed solve
        dict(name="sigma_mrcis_mixed_k8", do="sigma", prec="mixed", k=8, **_space("mrcis", 8, 6, 40)),
        # the same for a singles-and-doubles space in plain FP64
        dict(name="sigma_mrcisd_fp64_k8", do="sigma", prec="fp64", k=8, **_space("mrcisd", 8, 6, 24)),
        # odd electron count, 5 vectors: the float-float product of a refinement phase in which
        # some roots have converged
        dict(name="sigma_odd_ff_k5", do="sigma", prec="ff", k=5, **_space("mrcisd", 7, 5, 21, ksym=2)),
        # no stored matrix, two-word bit-strings (66 orbitals)
        dict(name="direct_mrcisd_k8", do="direct", prec="fp64", k=8, **_space("mrcisd", 6, 4, 60)),
        # valence full CI of 6 electrons in 12 orbitals
        dict(name="build_fci", do="build", prec="fp64", k=4, **_space("fci", 12, 6)),
        # the largest: about 2.2 million SEFs, built with the FP32 copy
        dict(name="build_mrcisd_large", do="build", prec="mixed", k=8, **_space("mrcisd", 8, 6, 48)),
        # up to 8 open shells (128 determinants a configuration)
        dict(name="build_open8", do="build", prec="fp64", k=4, **_space("fci", 10, 8)),
        # whole solves from new inputs: 4 roots tightly in FP64 with their vectors ...
        dict(name="solve_fci_fp64", do="solve", prec="fp64", k=4, rtol=1e-8, **_space("fci", 8, 6)),
        # ... and 8 roots in mixed precision, energies only
        dict(name="solve_mrcis_mixed", do="solve", prec="mixed", k=8, rtol=1e-5, **_space("mrcis", 8, 6, 40)),
        # properties of 8 roots
        dict(name="density_mrcisd_k8", do="density", prec="fp64", k=8, **_space("mrcisd", 8, 6, 24)),
        dict(name="gradient_mrcisd_k8", do="gradient", prec="fp64", k=8, nonzero=True, **_space("mrcisd", 8, 6, 16)),
    ]


def _log_int(rng, lo, hi):
    return min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49))))))


def draw(rng):
    """One more case: any call, space family, electron count, blocks of 2 to 8 vectors."""
    do = rng.choice(["sigma", "sigma", "build", "build", "direct", "solve", "density", "gradient"])
    kind = rng.choice(["fci", "mrcis", "mrcisd", "mrcisd"])
    if kind == "fci":
        nact, nelec = rng.choice([(8, 6), (9, 5), (9, 7), (10, 5), (10, 6), (10, 8), (11, 6), (12, 6)])
        nvirt = 0
        if do in ("direct", "gradient") and nelec > 6:  # more than a second
            nelec = 6
    else:
        nact, nelec = rng.choice([(5, 5), (6, 4), (6, 5), (6, 6), (7, 5), (7, 6), (8, 6)])
        most = 60 if kind == "mrcis" else {"gradient": 13, "direct": 24, "density": 32, "solve": 12}.get(do, 40)
        nvirt = _log_int(rng, 4, most)
    c = dict(do=do, k=rng.randint(2, 8), **_space(kind, nact, nelec, nvirt, ksym=rng.choice([1, 2])))
    c["prec"] = rng.choice({"sigma": ["fp64", "mixed", "mixed", "ff"], "build": ["fp64", "mixed", "mixed"],
                            "direct": ["fp64", "mixed"], "gradient": ["fp64", "mixed"]}.get(do, ["fp64"]))
    if do == "solve":
        c["prec"] = rng.choice(["fp64", "mixed"])
        c["rtol"] = 1e-8 if c["prec"] == "fp64" else 1e-5
    if do == "gradient":
        c["nonzero"] = rng.choice([True, False])
    return c


def _problem(case, seed):
    kw = dict(nact=case["nact"], nelec=case["nelec"], nvirt=case["nvirt"])
    if case["space"] == "fci":
        kw = dict(nbf=case["nact"], nelec=case["nelec"])
    return make_problem(case["space"], seed=seed, ksym=case["ksym"], **kw)


def _amplitudes(shape, seed):
    """CI-like coefficients: a few large ones and a long tail over six decades."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(shape, dtype=torch.float64, device="cuda", generator=g)
    return x * 10.0 ** (-6.0 * torch.rand(shape, dtype=torch.float64, device="cuda", generator=g) ** 2)


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case, p = case, _problem(case, seed)
    s.problem, s.one = p, p.one_packed()
    s.ctx = api.Context(0)
    if case["do"] == "solve":  # a kept context; everything else is the call's own work
        return s
    s.ctx.load_problem(p)
    n, k, do = p.num_sefs(), case["k"], case["do"]
    if do != "build":
        s.ctx.build_determinants()
    if do in ("sigma", "direct"):
        s.ctx.build_hamiltonian(mixed=case["prec"] == "mixed", direct=do == "direct")
    if do in ("sigma", "direct", "build"):  # one row per SEF, the block's vectors side by side
        s.x = _amplitudes((n, k), seed)
        s.y = torch.empty_like(s.x)
        return s
    s.x = _amplitudes((k, n), seed)  # one root after another
    s.x /= s.x.norm(dim=1, keepdim=True)
    n1 = p.nbf * (p.nbf + 1) // 2
    s.d1 = torch.empty((k, n1), dtype=torch.float64, device="cuda")
    if do == "gradient":
        s.d2 = torch.empty((k, n1 * (n1 + 1) // 2), dtype=torch.float64, device="cuda")
    return s


def run(s):
    c, ctx, p = s.case, s.ctx, s.problem
    do, k, prec = c["do"], c["k"], PREC[c["prec"]]
    if do == "solve":
        mixed = c["prec"] == "mixed"
        ctx.set_integrals(p.nbf, s.one, p.eri, p.ecore)
        ctx.set_configs(p.nbf, p.nelec, p.ksym, p.mx_open, p.jsym, p.occ)
        ctx.build_determinants()
        ctx.build_hamiltonian(mixed=mixed)
        r = ctx.davidson(k, rtol=c["rtol"], mixed=mixed, want_vectors=not mixed)
        return [r.evals] if mixed else [r.evals, r.evecs]
    if do == "density":
        ctx.density1_device(s.x.data_ptr(), s.x.shape[1], s.d1.data_ptr(), k)
        return s.d1
    if do == "gradient":
        ctx.energy_gradient_device(s.x.data_ptr(), s.x.shape[1], k, s.d1.data_ptr(), s.d2.data_ptr(),
                                   nonzero_only=c["nonzero"], prec=prec)
        return [s.d1, s.d2]
    if do == "build":
        ctx.build_determinants()
        ctx.build_hamiltonian(mixed=c["prec"] == "mixed")
    ctx.sigma_device(s.x.data_ptr(), k, s.y.data_ptr(), k, k, prec)
    return s.y


_nnz = {}


def _stored(case):
    """Elements that the block's matrix stores (of one seed's integrals; others differ little)."""
    key = tuple(case[q] for q in ("space", "nact", "nelec", "nvirt", "ksym"))
    if key not in _nnz:
        with api.Context(0) as ctx:
            ctx.load_problem(_problem(case, 1))
            ctx.build_determinants()
            _nnz[key] = ctx.build_hamiltonian(mixed=False)
    return _nnz[key]


def work(case):
    p = _problem(case, 1)
    n, k, do = p.num_sefs(), case["k"], case["do"]
    n1 = p.nbf * (p.nbf + 1) // 2
    ints = 8 * (n1 + n1 * (n1 + 1) // 2)
    inputs = ints + p.nconf * (p.nbf + 4)
    if do == "density":
        return {"bytes": inputs - ints + 8 * n * k + 8 * n1 * k, "flops": 2.0 * n * k}
    if do == "gradient":
        return {"bytes": inputs + 8 * n * k + ints * k, "flops": 2.0 * _stored(case) * k}
    nnz = _stored(case)
    if do == "direct":
        return {"bytes": inputs + 16 * n * k, "flops": 2.0 * nnz * k}
    elem = 4 + (4 if case["prec"] == "mixed" else 8)  # a column index and a value of the product's type
    product = elem * nnz + 8 * (n + 1) + 16 * n * k
    if do == "sigma":
        return {"bytes": product, "flops": 2.0 * nnz * k}
    written = (12 + (4 if case["prec"] == "mixed" else 0)) * nnz + 8 * (n + 1)
    return {"bytes": inputs + written + product, "flops": 2.0 * nnz * k}


# ----------------------------------------------------------------------------------
# the same in 64 bits, for blocks small enough to form densely: determinants, Slater-Condon
# rules on their occupation strings and the transformation to SEFs, in numpy alone
# ----------------------------------------------------------------------------------
MOST_DETS = 5000


def _templates(parity, odd_class, nopen):
    """(alpha, beta) patterns over the open shells, in the order that numbers the determinants."""
    full = (1 << nopen) - 1
    size = lambda k: [m for m in range(1 << nopen) if m.bit_count() == k]  # noqa: E731
    if parity:
        m, out = (nopen - 1) // 2, []
        for s in range(nopen - m):
            out += [(c, full ^ c) if (s % 2 == 0) != odd_class else (full ^ c, c) for c in size(m + 1 + s)]
        return out
    if nopen == 0:
        return [(0, 0)]
    m, out = nopen // 2, []
    for delta in range(1 if odd_class else 0, m + 1, 2):
        cs = size(m + delta)
        for c in cs[:len(cs) // 2] if delta == 0 else cs:
            out += [(c, full ^ c), (full ^ c, c)]
    return out


def _determinants(p):
    """Per determinant: alpha and beta strings, phase, configuration; and the SEFs as columns."""
    al, be, ph, cf, rows, cols, vals, nsef = [], [], [], [], [], [], [], 0
    for i in range(p.nconf):
        occ, js = p.occ[i], int(p.jsym[i])
        opens = [int(q) for q in np.nonzero(occ == 1)[0]]
        doubles = [int(q) for q in np.nonzero(occ == 2)[0]]
        dbl = sum(1 << q for q in doubles)
        phase = sum(d > q for q in opens for d in doubles) & 1
        odd_class = (((js + 1) // 2) % 2 == 0) if p.nelec % 2 else ((js + 1) // 2 != (p.ksym + 1) // 2)
        m = -1.0 if js % 2 != p.ksym % 2 else 1.0
        spread = lambda t: sum(1 << q for b, q in enumerate(opens) if t >> b & 1)  # noqa: E731
        for d, (a, b) in enumerate(_templates(p.nelec % 2, odd_class, len(opens))):
            pair = p.nelec % 2 == 0 and bool(opens)
            if not pair or d % 2 == 0:
                nsef += 1
            rows.append(len(al))
            cols.append(nsef - 1)
            vals.append((math.sqrt(0.5) * (m if d % 2 else 1.0)) if pair else 1.0)
            al.append(dbl | spread(a))
            be.append(dbl | spread(b))
            ph.append(phase)
            cf.append(i)
    T = np.zeros((len(al), nsef))
    T[rows, cols] = vals
    return np.array(al, np.uint64), np.array(be, np.uint64), np.array(ph), np.array(cf), T


def _low_bit(x):
    return np.bitwise_count((x & (~x + np.uint64(1))) - np.uint64(1)).astype(np.int64)


def _between(string, p, q):
    """Electrons of `string` strictly between orbitals p and q."""
    one = np.uint64(1)
    lo, hi = np.minimum(p, q).astype(np.uint64), np.maximum(p, q).astype(np.uint64)
    return np.bitwise_count(string & ((one << hi) - one) & ~((one << (lo + one)) - one)).astype(np.int64)


def _dense(p):
    """H over the SEFs, with elements below the 1e-8 that storage keeps left out."""
    al, be, ph, cf, T = _determinants(p)
    nbf, one1 = p.nbf, p.one_packed()
    idx = np.arange(nbf)
    tri = lambda i, j: np.maximum(i, j) * (np.maximum(i, j) + 1) // 2 + np.minimum(i, j)  # noqa: E731
    h = one1[tri(idx[:, None], idx[None, :])]
    pq = tri(idx[:, None], idx[None, :])
    g = p.eri[tri(pq[:, :, None, None], pq[None, None, :, :])]
    bits = lambda s: ((s[:, None] >> idx.astype(np.uint64)) & np.uint64(1)).astype(np.float64)  # noqa: E731
    oa, ob = bits(al), bits(be)
    J, K = np.einsum("iijj->ij", g), np.einsum("ijij->ij", g)
    nd = len(al)
    H = np.zeros((nd, nd))
    n = oa + ob
    np.fill_diagonal(H, n @ np.diag(h) + 0.5 * (np.einsum("di,ij,dj->d", n, J, n) -
                                                np.einsum("di,ij,dj->d", oa, K, oa) - np.einsum("di,ij,dj->d", ob, K, ob)))
    js = p.jsym.astype(np.int64)
    na = np.bitwise_count(al).astype(np.int64)
    for r in range(nd):
        c = np.nonzero(cf <= cf[r])[0]  # the lower blocks; the others mirror them
        c = c[c != r]
        xa, ya, xb, yb = al[r] & ~al[c], al[c] & ~al[r], be[r] & ~be[c], be[c] & ~be[r]
        ka, kb = np.bitwise_count(ya).astype(np.int64), np.bitwise_count(yb).astype(np.int64)
        differ = np.bitwise_count(xa).astype(np.int64) + np.bitwise_count(xb).astype(np.int64)
        sym = js[cf[c]] == js[cf[r]]
        sign = 1.0 - 2.0 * ((ph[r] + ph[c]) & 1)
        same = na[c] == na[r]
        one_conf = np.bitwise_count((al[r] | be[r]) ^ (al[c] | be[c])) + np.bitwise_count((al[r] & be[r]) ^ (al[c] & be[c])) == 2
        # one electron moved within its spin, equal symmetries
        t = np.nonzero(same & (differ == 1) & sym & (ka + kb == 1))[0]
        if len(t):
            alpha = ka[t] == 1
            i, j = _low_bit(np.where(alpha, xa[t], xb[t])), _low_bit(np.where(alpha, ya[t], yb[t]))
            own = np.where(alpha[:, None], oa[r][None], ob[r][None])
            v = h[i, j] + np.einsum("tr,r->t", g[i, j][:, idx, idx], n[r]) - np.einsum("tr,tr->t", g[i, :, :, j][:, idx, idx], own)
            flips = _between(np.where(alpha, al[r], be[r]), i, j)
            H[r, c[t]] = v * sign[t] * (1 - 2 * (flips & 1))
        # spin-orbit: one electron moved, any spins, unequal symmetries
        t = np.nonzero((differ == 1) & ~sym & one_conf)[0]
        if len(t):
            i, j = _low_bit(xa[t] | xb[t]), _low_bit(ya[t] | yb[t])
            v = 0.5 * h[i, j] * np.where(j > i, -1.0, 1.0)
            jr, jc, o = js[cf[r]], js[cf[c[t]]], np.uint64(1)
            iu, ju, top = i.astype(np.uint64), j.astype(np.uint64), ~np.uint64(0)
            below = lambda q: (o << q) - o  # noqa: E731
            above = lambda q: top & ~((o << (q + o)) - o)  # noqa: E731
            up = np.bitwise_count(be[r] & below(iu)) + np.bitwise_count(al[c[t]] & above(ju)) + np.where((jr + jc) % 2 == 0, 1, jr % 2)
            down = np.bitwise_count(al[r] & above(iu)) + np.bitwise_count(be[c[t]] & below(ju)) + (((jr + jc) % 2) & (jr % 2))
            beta = ka[t] == 0
            kept = beta + jr % 2 + _between(np.where(beta, be[r], al[r]), i, j)
            f = np.where(na[r] < na[c[t]], up, np.where(na[r] > na[c[t]], down, kept)).astype(np.int64)
            H[r, c[t]] = v * sign[t] * (1 - 2 * (f & 1))
        # two electrons of opposite spin
        t = np.nonzero(same & (ka == 1) & (kb == 1))[0]
        if len(t):
            i, j, k, l = _low_bit(xa[t]), _low_bit(ya[t]), _low_bit(xb[t]), _low_bit(yb[t])
            flips = _between(np.broadcast_to(al[r], t.shape), i, j) + _between(np.broadcast_to(be[r], t.shape), k, l)
            H[r, c[t]] = g[i, j, k, l] * sign[t] * (1 - 2 * (flips & 1))
        # two electrons of one spin
        t = np.nonzero(same & (ka + kb == 2) & ((ka == 2) | (kb == 2)))[0]
        if len(t):
            alpha = ka[t] == 2
            x, y = np.where(alpha, xa[t], xb[t]), np.where(alpha, ya[t], yb[t])
            i0, j0 = _low_bit(x), _low_bit(y)
            i1, j1 = _low_bit(x & (x - np.uint64(1))), _low_bit(y & (y - np.uint64(1)))
            s, u = np.where(alpha, al[r], be[r]), np.where(alpha, al[c[t]], be[c[t]])
            flips = _between(s, i0, i1) + _between(u, j0, j1)
            H[r, c[t]] = (g[i0, j0, i1, j1] - g[i0, j1, i1, j0]) * sign[t] * (1 - 2 * (flips & 1))
    H = np.where(cf[:, None] >= cf[None, :], H, 0.0)
    H = T.T @ H @ T
    H = np.tril(H) + np.tril(H, -1).T
    return np.where((np.abs(H) >= 1e-8) | np.eye(len(H), dtype=bool), H, 0.0)


def exact(case, seed):
    """H X, or the lowest eigenvalues, of a block of at most 5000 determinants; larger blocks and
    the densities would take a second Slater-Condon engine more than 20 seconds."""
    if case["do"] not in ("sigma", "direct", "build", "solve"):
        return None
    p = _problem(case, seed)
    if int(p.ndet().sum()) > MOST_DETS or p.nbf > 62:  # strings of one 64-bit word
        return None
    H = _dense(p)
    if case["do"] == "solve":
        w = np.linalg.eigvalsh(H)[:case["k"]]
        return [w] if case["prec"] == "mixed" else [w, None]
    return H @ _amplitudes((len(H), case["k"]), seed).cpu().numpy()
