"""Performance cases of the selected-CI path: the calls that a user's program
makes into macis_b200, over the sizes that it makes them at.

A case is a dict of plain values. ``op`` names the call:

* ``cas_solve``  selected_ci_diag on a full CAS space (build + Davidson)
* ``cas_build``  CSR build of a CAS space on device determinants, one product
* ``sel_build``  the same on a selected (ASCI-shaped) determinant list
* ``sel_solve``  selected_ci_diag on a selected list
* ``hop``        one product of a matrix-free Hamiltonian that is kept
* ``rdm``        form_rdms of a CAS or selected wavefunction
* ``search``     asci_search (exact)
* ``screen``     asci_search with the network pruning the units
* ``train``      the network's training on the samples of a search

Integrals follow the repository's synthetic recipe (orbital energies on a
ramp, weak off-diagonal one-body terms, two-body terms as sums of products of
symmetric factors). Selected lists are excitations of degree 0 to 4 from the
lowest determinant that prefer the orbitals near the Fermi level, ordered as a
search returns them: new determinants ascending, then the core determinants.
"""
import itertools
import math

import numpy as np
import torch

import macis_b200 as mb
from macis_b200 import _lib
from macis_b200._lib import LIB, check

EPS = float(np.finfo(np.float64).eps)
DAV = dict(restart_keep=8, max_iter=4000)   # thick restart, as the benchmark


def listed():
    return [
        # the first steps of a grow: a space of a few hundred determinants,
        # where launches, synchronisations and allocations are all there is
        dict(name="cas_solve_6o", op="cas_solve", n=6, ka=3, kb=3, prec="fp64"),
        # a CAS solve of ordinary size, FP32-stored H (63,504 determinants)
        dict(name="cas_solve_10o_mixed", op="cas_solve", n=10, ka=5, kb=5,
             prec="mixed"),
        # the largest full CI of the benchmark (853,776 determinants)
        dict(name="cas_build_12o", op="cas_build", n=12, ka=6, kb=6,
             prec="fp64"),
        # H of an ASCI wavefunction, bitset<128>
        dict(name="sel_build_n48", op="sel_build", n=48, k=12, nbits=128,
             ndets=150001, prec="fp64"),
        # rediagonalisation in the middle of a grow, bitset<64>
        dict(name="sel_solve_n24", op="sel_solve", n=24, k=6, nbits=64,
             ndets=20011, prec="fp64"),
        # H x without storing H, the operator of the lists that do not fit
        dict(name="hop_n64_mixed", op="hop", n=64, k=16, nbits=128,
             ndets=100003, prec="mixed"),
        # density matrices of a CAS wavefunction
        dict(name="rdm_cas_9o", op="rdm", space="cas", n=9, ka=4, kb=4,
             two=True),
        # a search from a small core set (grow start)
        dict(name="search_n48_small", op="search", n=48, k=12, nbits=128,
             ncore=50, ndets=20000),
        # a search of a refine iteration at ordinary size
        dict(name="search_n48", op="search", n=48, k=12, nbits=128,
             ncore=10000, ndets=200000),
        # the widest determinants, 100 orbitals in bitset<256>
        dict(name="search_n100", op="search", n=100, k=20, nbits=256,
             ncore=301, ndets=6020),
        # a search pruned by the network (forward over all units)
        dict(name="screen_n48", op="screen", n=48, k=12, nbits=128,
             ncore=5003, ndets=100000),
        # the training after a recording search
        dict(name="train_n48", op="train", n=48, k=12, nbits=128, ncore=150,
             samples=131072, epochs=2, batch=1024),
    ]


def _log(rng, lo, hi):
    """A whole number, evenly spread over the logarithm of [lo, hi]."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["cas_solve", "cas_build", "sel_build", "sel_solve", "hop",
                     "rdm", "search", "search", "screen", "train"])
    prec = rng.choice(["fp64", "mixed"])
    nbits = rng.choice([64, 128])
    if op in ("cas_solve", "cas_build"):
        n = rng.randint(6, 10 if op == "cas_solve" else 11)
        return dict(op=op, n=n, ka=rng.randint(2, n // 2),
                    kb=rng.randint(2, n // 2), prec=prec)
    if op == "rdm":
        if rng.random() < 0.5:
            n = rng.randint(6, 9)
            return dict(op=op, space="cas", n=n, ka=rng.randint(2, n // 2),
                        kb=rng.randint(2, n // 2), two=rng.random() < 0.75)
        n = rng.randint(16, 32)
        return dict(op=op, space="sel", n=n, k=rng.randint(4, 7), nbits=nbits,
                    ndets=_log(rng, 500, 15000), two=rng.random() < 0.75)
    if op in ("sel_build", "sel_solve", "hop"):
        n = rng.randint(16, 32) if nbits == 64 else rng.randint(33, 64)
        top = {"sel_build": 150000, "sel_solve": 30000, "hop": 100000}[op]
        return dict(op=op, n=n, k=rng.randint(5, n // 4 + 1), nbits=nbits,
                    ndets=_log(rng, 500, top), prec=prec)
    if op == "train":
        return dict(op=op, n=48, k=12, nbits=128, ncore=rng.randint(40, 150),
                    samples=_log(rng, 4000, 131072), epochs=rng.randint(1, 2),
                    batch=rng.choice([256, 1000, 1024, 4096]))
    nbits = rng.choice([64, 128, 128, 256]) if op == "search" else 128
    n = {64: rng.randint(16, 32), 128: rng.randint(33, 64),
         256: rng.randint(66, 100)}[nbits]
    k = rng.randint(5, n // 5 + 2)
    # contributions of one core determinant, to stay below the largest case
    per = k * (n - k) * (2 + k * (n - k)) + 2 * math.comb(k, 2) * math.comb(n - k, 2)
    top = max(40, min(10000, int(2.4e9 / per)))
    nc = _log(rng, 20, top if op == "search" else max(40, top // 2))
    return dict(op=op, n=n, k=k, nbits=nbits, ncore=nc,
                ndets=nc * rng.randint(8, 40))


# ------------------------------------------------------------------- inputs
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _gen(seed, salt):
    g = torch.Generator(device=_dev())
    g.manual_seed(1000003 * int(seed) + salt)
    return g


def integrals(n, seed):
    """(T, V) flat column-major: the synthetic recipe, with the 8-fold
    symmetry exact (V is computed for the packed pairs p <= q)."""
    d, g = _dev(), _gen(seed, 1)
    eps = -1.5 + 2.5 * torch.arange(n, dtype=torch.float64, device=d) / max(n - 1, 1)
    off = torch.triu(0.02 * torch.randn(n, n, dtype=torch.float64, device=d,
                                        generator=g), 1)
    T = off + off.T + torch.diag(eps)
    ip, iq = torch.triu_indices(n, n, device=d)
    scale = 0.3 * torch.exp(-torch.arange(2 * n, dtype=torch.float64, device=d) / n)
    B = scale[:, None] * torch.randn(2 * n, len(ip), dtype=torch.float64,
                                     device=d, generator=g)
    P = B.T @ B
    P = torch.triu(P) + torch.triu(P, 1).T
    pair = torch.empty(n, n, dtype=torch.int64, device=d)
    at = torch.arange(len(ip), device=d)
    pair[ip, iq] = at
    pair[iq, ip] = at
    pair = pair.reshape(-1)
    V = P[pair][:, pair].reshape(-1)        # symmetric: any index order
    return T.reshape(-1).cpu().numpy(), V.cpu().numpy()


def _words(mask):
    """uint64 words (as int64) of boolean occupations [N, n], 64 per word."""
    out = []
    for lo in range(0, mask.shape[1], 64):
        m = mask[:, lo:lo + 64].to(torch.int64)
        out.append((m << torch.arange(m.shape[1], device=m.device)).sum(1))
    return out


def _window(n, k, ndets):
    """Holes and particles around the Fermi level that a list of ndets
    determinants uses: about 20 times as many excitations of degree <= 4, so
    that each determinant has its neighbours in the list, as one that a
    search selected has."""
    for m in range(2, n):
        h, p = min(k, m), min(n - k, 2 * m)
        links = [math.comb(h, e) * math.comb(p, e) for e in range(5)]
        if sum(links[e] * links[f] for e in range(5) for f in range(5 - e)) >= 20 * ndets:
            break
    return h, p


def _excite(n, k, deg, h, p, g):
    """Occupations of the lowest-k string with deg[i] electrons moved from
    the last h occupied to the first p empty orbitals, those near the Fermi
    level preferred."""
    d, N = deg.device, len(deg)

    def pick(size, use):                    # the first `use` of `size`
        near = torch.arange(size, dtype=torch.float64, device=d)
        key = torch.rand(N, size, generator=g, device=d, dtype=torch.float64)
        key = -torch.log(-torch.log(key.clamp(1e-12, 1 - 1e-12))) - near / use
        key = torch.where(near < use, key, key - 1e6)
        rank = torch.argsort(torch.argsort(-key, dim=1), dim=1)
        return rank < deg[:, None]
    return torch.cat([~pick(k, h).flip(1), pick(n - k, p)], 1)


def selected(n, k, nbits, ndets, seed, weights=(0.02, 0.18, 0.3, 0.5)):
    """ndets determinants by ascending excitation degree (random inside one
    degree), the lowest determinant first; uint64 [ndets, nbits // 64]."""
    d, g = _dev(), _gen(seed, 2)
    w = torch.tensor(weights, dtype=torch.float64, device=d)
    h, p = _window(n, k, ndets)
    got = torch.zeros(0, 1 + nbits // 64, dtype=torch.int64, device=d)
    for _ in range(12):
        N = 2 * ndets + 64
        tot = 1 + torch.multinomial(w, N, replacement=True, generator=g)
        tot[0] = 0
        ea = (torch.rand(N, 4, generator=g, device=d) < 0.5)
        ea = (ea & (torch.arange(4, device=d)[None] < tot[:, None])).sum(1)
        eb = (tot - ea).clamp(max=h)
        ea = ea.clamp(max=h)
        tot = ea + eb
        a = _words(_excite(n, k, ea, h, p, g))
        b = _words(_excite(n, k, eb, h, p, g))
        if nbits == 64:
            words = [a[0] | (b[0] << 32)]
        elif nbits == 128:
            words = [a[0], b[0]]
        else:
            z = torch.zeros_like(a[0])
            words = (a + [z])[:2] + (b + [z])[:2]
        got = torch.unique(torch.cat([got, torch.stack([tot] + words, 1)]), dim=0)
        if len(got) >= ndets:
            break
    # a sample of the right size, the lowest determinant always in it
    keep = torch.randperm(len(got) - 1, generator=g, device=d)[:ndets - 1] + 1
    got = torch.cat([got[:1], got[keep]])
    order = torch.sort(got[:, 0], stable=True).indices
    return got[order, 1:].cpu().numpy().view(np.uint64)


def search_order(dets, ncore):
    """New determinants ascending, then the leading ncore ones."""
    core, new = dets[:ncore], dets[ncore:]
    new = new[np.lexsort(tuple(new[:, j] for j in range(new.shape[1])))]
    return np.ascontiguousarray(np.concatenate([new, core]))


def coefficients(m, seed):
    """Normalised coefficients in decreasing magnitude, random signs."""
    rng = np.random.default_rng([int(seed), 3])
    c = (1.0 + np.arange(m)) ** -0.75 * np.exp(0.3 * rng.standard_normal(m))
    c = -np.sort(-c) * rng.choice([-1.0, 1.0], m)
    return c / np.linalg.norm(c)


def _occ(n, k):
    return np.array(list(itertools.combinations(range(n), k)), dtype=np.int64)


def cas(n, ka, kb):
    """All determinants, alpha outer, strings by ascending occupied tuple."""
    a = (np.uint64(1) << _occ(n, ka).astype(np.uint64)).sum(1, dtype=np.uint64)
    b = (np.uint64(1) << _occ(n, kb).astype(np.uint64)).sum(1, dtype=np.uint64)
    return (a[:, None] | (b[None] << np.uint64(32))).reshape(-1, 1)


def _vector(m, seed):
    return torch.randn(m, dtype=torch.float64, device=_dev(),
                       generator=_gen(seed, 4))


def _case_dets(case, seed):
    if case["op"].startswith("cas") or case.get("space") == "cas":
        return cas(case["n"], case["ka"], case["kb"])
    d = selected(case["n"], case["k"], case["nbits"], case["ndets"], seed)
    return search_order(d, max(1, len(d) // 10))


def prepare(case, seed):
    op, n = case["op"], case["n"]
    T, V = integrals(n, seed)
    H = mb.HamiltonianGenerator(T, V, case.get("nbits", 64))
    s = dict(case=case, H=H)
    vt = np.float32 if case.get("prec") == "mixed" else np.float64
    if op in ("search", "screen", "train"):
        core = selected(n, case["k"], case["nbits"], case["ncore"], seed,
                        weights=(0.1, 0.5, 0.25, 0.15))
        s.update(core=core, C=coefficients(len(core), seed),
                 E0=float(H.matrix_element(core[:1], core[:1])) - 0.5,
                 asci=mb.ASCISettings())
        if op == "screen":
            s["net"] = _network(case["nbits"], seed)
        elif op == "train":
            s["net"] = mb.ScreeningNetwork(nbits=case["nbits"], seed=seed)
            rec = mb.ScreenSettings(network=s["net"], seed=seed,
                                    max_samples=case["samples"])
            mb.asci_search(s["asci"], 20 * len(core), core, s["E0"], s["C"], n,
                           H, screen=rec)
            s["net"].clamp_samples(rec.clamp_quantile)
        return s
    dets = _case_dets(case, seed)
    s["dets"] = dets
    if op in ("cas_build", "sel_build", "hop"):
        s["x"] = _vector(len(dets), seed)
        s["y"] = torch.zeros_like(s["x"])
        s["value_t"] = vt
        if op == "hop":
            s["op"] = mb.MatrixFreeHamiltonian(dets, H, EPS, value_t=vt)
        else:
            s["ddets"] = torch.from_numpy(dets.view(np.int64)).to(_dev())
    elif op == "rdm":
        c = coefficients(len(dets), seed)
        # a CAS vector has its large coefficients anywhere in the list
        s["C"] = np.random.default_rng([int(seed), 5]).permutation(c)
    return s


def _network(nbits, seed):
    """A network that ranks units by the crude log-score estimate among its
    inputs, perturbed by small random weights."""
    net = mb.ScreeningNetwork(nbits=nbits, seed=seed)
    p = net.params * np.float32(0.05)
    din, h = net.din, 256
    w2 = h * din + h
    w3 = w2 + h * h + h
    p[din - 64 + 15] = 1.0                  # W1[0, estimate]
    p[h * din] = 4.0                        # b1[0]
    p[w2] = 1.0                             # W2[0, 0]
    p[w3] = 1.0                             # w3[0]
    net.params = p
    return net


# --------------------------------------------------------------------- runs
def run(s):
    c, H = s["case"], s["H"]
    op = c["op"]
    if op in ("cas_solve", "sel_solve"):
        E, X = mb.selected_ci_diag(
            s["dets"], H, EPS, 40, 1e-8, index_t=None,
            precision=mb.MIXED if c["prec"] == "mixed" else mb.FP64, **DAV)
        return {"E": E, "X": X}
    if op in ("cas_build", "sel_build"):
        A = mb.make_csr_hamiltonian(s["ddets"], H, EPS, value_t=s["value_t"])
        check(LIB.macis_b200_spmv(A.handle, 1, 1.0, s["x"].data_ptr(), A.n, 0.0,
                                  s["y"].data_ptr(), A.m, _lib.DEVICE_PTRS))
        return {"nnz": A.nnz, "y": s["y"]}
    if op == "hop":
        A = s["op"]
        check(LIB.macis_b200_hop_apply(A.handle, 1, 1.0, s["x"].data_ptr(), A.n,
                                       0.0, s["y"].data_ptr(), A.m,
                                       _lib.DEVICE_PTRS))
        return {"y": s["y"]}
    if op == "rdm":
        ordm, trdm = H.form_rdms(s["dets"], s["C"], two=c["two"])
        return {"ordm": ordm} if trdm is None else {"ordm": ordm, "trdm": trdm}
    if op == "search":
        return mb.asci_search(s["asci"], c["ndets"], s["core"], s["E0"], s["C"],
                              c["n"], H)
    if op == "screen":
        scr = mb.ScreenSettings(network=s["net"], keep_frac=0.2,
                                explore_frac=0.02, train=False)
        return mb.asci_search(s["asci"], c["ndets"], s["core"], s["E0"], s["C"],
                              c["n"], H, screen=scr, use_net=True)
    if op == "train":
        loss = s["net"].train(None, None, c["epochs"], c["batch"], 1e-3, 7)
        return {"loss": loss, "params": s["net"].params}
    raise ValueError(op)


# --------------------------------------------------------------------- work
def _string_links(n, k):
    """(singles, doubles) of one string."""
    return k * (n - k), math.comb(k, 2) * math.comb(n - k, 2)


def work(case):
    """Determinants, integrals and vectors read and written once, a stored
    matrix written once, and two operations for every matrix element or
    contribution that the exact counts give (selected lists: the diagonal and
    the vectors alone, since their element count depends on the list)."""
    op, n = case["op"], case["n"]
    nw = case.get("nbits", 64) // 64
    ints = 8.0 * (n ** 4 + n ** 2)
    if op in ("cas_solve", "cas_build") or case.get("space") == "cas":
        sa, da = _string_links(n, case["ka"])
        sb, db = _string_links(n, case["kb"])
        N = math.comb(n, case["ka"]) * math.comb(n, case["kb"])
        nnz = float(N) * (1 + sa + sb + da + db + sa * sb)
        if op == "rdm":
            out = 8.0 * (n * n + (n ** 4 if case["two"] else 0))
            return {"bytes": 16.0 * N + out, "flops": 8 * nnz if case["two"] else 2.0 * N * (sa + sb)}
        val = 4 if case["prec"] == "mixed" else 8
        return {"bytes": ints + 16.0 * N + nnz * (4 + val), "flops": 2 * nnz}
    if op in ("sel_build", "sel_solve", "hop", "rdm"):
        N = case["ndets"]
        out = 8.0 * n ** 4 if op == "rdm" else ints
        return {"bytes": out + N * (8.0 * nw + 16), "flops": 2.0 * N}
    if op == "train":
        rows = float(case["samples"]) * case["epochs"]
        return {"bytes": rows * 388, "flops": rows * 3 * 2 * (192 * 256 + 256 * 256 + 256)}
    s1, d1 = _string_links(n, case["k"])
    pairs = float(case["ncore"]) * (2 * s1 + 2 * d1 + s1 * s1)
    units = float(case["ncore"]) * (2 + 3 * s1)
    b = ints + 8.0 * nw * (case["ncore"] + case["ndets"])
    if op == "screen":
        return {"bytes": b, "flops": 0.22 * 20 * pairs + 229888 * units}
    return {"bytes": b, "flops": 20 * pairs}


# -------------------------------------------------------------------- exact
def exact(case, seed):
    """What run() computes, in 64 bits with torch: products and density
    matrices of CAS spaces from excitation operators on the CI vector, the
    lowest eigenvalue of small CAS spaces. The other outputs are whole
    numbers, eigenvectors stopped at a residual, or products over lists that
    only a pair search would give."""
    op = case["op"]
    if op == "cas_build":
        T, V = integrals(case["n"], seed)
        ops = _Excitations(case["n"], case["ka"], case["kb"])
        y = ops.product(T, V, _vector(ops.na * ops.nb, seed).reshape(ops.na, ops.nb))
        return {"nnz": None, "y": y.reshape(-1)}
    if op == "rdm" and case["space"] == "cas" and case["two"]:
        ops = _Excitations(case["n"], case["ka"], case["kb"])
        c = coefficients(ops.na * ops.nb, seed)
        c = np.random.default_rng([int(seed), 5]).permutation(c)
        ordm, trdm = ops.density(torch.from_numpy(c).to(_dev()).reshape(ops.na, ops.nb))
        return {"ordm": ordm.cpu().numpy(), "trdm": trdm.cpu().numpy()}
    if op == "cas_solve" and case["prec"] == "fp64":
        N = math.comb(case["n"], case["ka"]) * math.comb(case["n"], case["kb"])
        if N <= 1500:
            T, V = integrals(case["n"], seed)
            ops = _Excitations(case["n"], case["ka"], case["kb"])
            eye = torch.eye(N, dtype=torch.float64, device=_dev())
            Hm = torch.stack([ops.product(T, V, e.reshape(ops.na, ops.nb)).reshape(-1)
                              for e in eye])
            return {"E": float(torch.linalg.eigvalsh(0.5 * (Hm + Hm.T))[0]), "X": None}
    return None


class _Excitations:
    """E_pq = a+_p a_q summed over spin, on CI vectors [alpha, beta] of a
    full CAS space in the order of cas()."""

    def __init__(self, n, ka, kb):
        self.n = n
        self.a, self.na = self._table(n, ka)
        self.b, self.nb = self._table(n, kb)

    @staticmethod
    def _table(n, k):
        """Per (p, q): source strings, target strings, signs."""
        occ = _occ(n, k)
        index = {tuple(o): i for i, o in enumerate(occ)}
        table = {}
        for i, o in enumerate(occ):
            o = tuple(int(x) for x in o)
            for q in o:
                rest = tuple(x for x in o if x != q)
                sq = sum(x < q for x in o)
                for p in range(n):
                    if p in rest:
                        continue
                    sp = sum(x < p for x in rest)
                    j = index[tuple(sorted(rest + (p,)))]
                    table.setdefault((p, q), []).append((i, j, -1.0 if (sq + sp) & 1 else 1.0))
        d = _dev()
        return {pq: (torch.tensor([t[0] for t in v], device=d),
                     torch.tensor([t[1] for t in v], device=d),
                     torch.tensor([t[2] for t in v], dtype=torch.float64, device=d))
                for pq, v in table.items()}, len(occ)

    def apply(self, p, q, x):
        y = torch.zeros_like(x)
        if (p, q) in self.a:
            src, dst, sg = self.a[p, q]
            y[dst] += sg[:, None] * x[src]
        if (p, q) in self.b:
            src, dst, sg = self.b[p, q]
            y[:, dst] += sg * x[:, src]
        return y

    def product(self, T, V, x):
        """H x = sum_pq E_pq (h_pq x + 1/2 sum_rs (pq|rs) E_rs x), with h_pq
        = T_pq - 1/2 sum_r (pr|rq)."""
        n, d = self.n, x.device
        V4 = torch.from_numpy(V).to(d).reshape(n, n, n, n)
        h = torch.from_numpy(T).to(d).reshape(n, n) - 0.5 * torch.einsum("prrq->pq", V4)
        M = torch.stack([self.apply(r, s, x).reshape(-1)
                         for r in range(n) for s in range(n)])
        W = 0.5 * V4.reshape(n * n, n * n)
        y = torch.zeros_like(x)
        for p in range(n):
            for q in range(n):
                z = (W[p * n + q] @ M).reshape(x.shape) + h[p, q] * x
                y += self.apply(p, q, z)
        return y

    def density(self, x):
        """ordm[p, q] = <E_pq>, trdm[p, q, r, s] = 1/2 (<E_pq E_rs> -
        delta_qr <E_ps>), where form_rdms, as the reference, keeps the
        same-spin exchange of a determinant with itself at (p, q, p, q)."""
        n = self.n
        M = torch.stack([self.apply(p, q, x).reshape(-1)
                         for p in range(n) for q in range(n)])
        one = (M @ x.reshape(-1)).reshape(n, n)
        # <E_pq E_rs> = (E_qp x) . (E_rs x)
        two = (M @ M.T).reshape(n, n, n, n).permute(1, 0, 2, 3).clone()
        for q in range(n):
            two[:, q, q, :] -= one
        w2, j = x * x, torch.arange(n, device=x.device)
        both = torch.zeros(n, n, dtype=x.dtype, device=x.device)
        for table, weight in ((self.a, w2.sum(1)), (self.b, w2.sum(0))):
            occ = torch.zeros(n, len(weight), dtype=x.dtype, device=x.device)
            for p in range(n):
                if (p, p) in table:
                    occ[p, table[p, p][0]] = 1.0
            both += (occ * weight) @ occ.T
        both.fill_diagonal_(0.0)
        p, q = j[:, None], j[None]
        two[p, q, q, p] += both
        two[p, q, p, q] -= both
        return one, 0.5 * two
