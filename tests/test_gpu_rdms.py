"""1- and 2-RDMs (macis_b200_form_rdms) against the reference's own
DoubleLoopHamiltonianGenerator::form_rdms (double_loop.hpp:117-165),
compiled here: sums are atomic on the GPU, so the tolerance is 1e-12
(absolute, the RDM entries are O(1))."""
import numpy as np
import pytest

import macis_b200 as mb
from cases import fci, shuffled

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nbits", [64, 128])
def test_rdms_match_reference(ref, nbits):
    T, V, d = fci(7, 3, 3, nbits, seed=2)
    sel = shuffled(d, seed=3, frac=0.7).copy()
    sel[9] = 0                                  # zero determinant: skipped
    sel[20] = sel[21]                           # duplicate determinant
    C = np.random.default_rng(1).standard_normal(len(sel))
    C /= np.linalg.norm(C)
    C[5] = 1e-17                                # pairs below 1e-16 skipped
    H = mb.HamiltonianGenerator(T, V, nbits)
    hr = ref.ham(nbits, 7, T, V)
    for two in (True, False):
        o, t = H.form_rdms(sel, C, two=two)
        ro, rt = ref.form_rdms(hr, sel, C, two=two)
        np.testing.assert_allclose(o.ravel(order="F"), ro, rtol=0,
                                   atol=1e-12)
        if two:
            np.testing.assert_allclose(t.ravel(order="F"), rt, rtol=0,
                                       atol=1e-12)


def test_rdm_traces_and_energy(port):
    """Tr(1-RDM) = electrons; E = sum h D1 + 1/2 sum V D2 for the ground
    state (the reference's RDM-energy identity, cas.hpp)."""
    T, V, d = fci(6, 3, 2, 64, seed=4)
    H = mb.HamiltonianGenerator(T, V, 64)
    E, X = mb.selected_ci_diag(d, H, np.finfo(float).eps, 60, 1e-10)
    o, t = H.form_rdms(d, X)
    assert abs(np.trace(o) - 5) < 1e-10
    n = 6
    Tm = np.asarray(T).reshape(n, n, order="F")
    Vm = np.asarray(V).reshape(n, n, n, n, order="F")
    E_rdm = np.einsum("pq,pq", Tm, o) + np.einsum("pqrs,pqrs", Vm, t)
    assert abs(E_rdm - E) < 1e-8


def _rdms_by_pairs(dets, C, n, two):
    """rdm_contributions (include/macis/util/rdms.hpp:15-131) summed over all
    pairs in plain Python, bra = ket = dets."""
    def between(s, x, y):
        lo, hi = min(x, y), max(x, y)
        return bin(s >> (lo + 1) & ((1 << max(hi - lo - 1, 0)) - 1)).count("1")

    def excite(bra, ket, k):  # k excitations: ((o, v), ...), sign
        ops, sg = [], 1
        for _ in range(k):
            x = bra ^ ket
            o = (ket & x) & -(ket & x)
            v = (bra & x) & -(bra & x)
            oi, vi = o.bit_length() - 1, v.bit_length() - 1
            sg *= -1 if between(ket, vi, oi) & 1 else 1
            ops.append((oi, vi))
            ket ^= o | v
        return ops, sg
    bits = lambda s: [p for p in range(n) if s >> p & 1]
    al, be = mb.sd.split_dets(dets, 64 * dets.shape[1])
    D1, D2 = np.zeros((n, n)), np.zeros((n, n, n, n))
    for i, (ba, bb) in enumerate(zip(al, be)):
        for j, (ka, kb) in enumerate(zip(al, be)):
            ca, cb = bin(ba ^ ka).count("1"), bin(bb ^ kb).count("1")
            val = C[i] * C[j]
            if ca + cb > 4 or not abs(val) > 1e-16 or not (ba or bb) or not (ka or kb):
                continue
            if (ca == 4 or cb == 4) and two:
                ((o1, v1), (o2, v2)), sg = excite(*((ba, ka) if ca == 4 else (bb, kb)), 2)
                v = 0.5 * sg * val
                D2[v1, o1, v2, o2] += v
                D2[v2, o1, v1, o2] -= v
                D2[v1, o2, v2, o1] -= v
                D2[v2, o2, v1, o1] += v
            elif ca == 2 and cb == 2 and two:
                ((oa, va),), sa = excite(ba, ka, 1)
                ((ob, vb),), sb = excite(bb, kb, 1)
                v = 0.5 * sa * sb * val
                D2[va, oa, vb, ob] += v
                D2[vb, ob, va, oa] += v
            elif ca == 2 or cb == 2:
                s, o = (ba, bb) if ca == 2 else (bb, ba)
                ((o1, v1),), sg = excite(*((ba, ka) if ca == 2 else (bb, kb)), 1)
                D1[v1, o1] += sg * val
                if two:
                    v = 0.5 * sg * val
                    for p in bits(s):
                        D2[v1, o1, p, p] += v
                        D2[p, p, v1, o1] += v
                        D2[v1, p, p, o1] -= v
                        D2[p, o1, v1, p] -= v
                    for p in bits(o):
                        D2[v1, o1, p, p] += v
                        D2[p, p, v1, o1] += v
            else:
                for p in bits(ba) + bits(bb):
                    D1[p, p] += val
                if two:
                    v = 0.5 * val
                    for s in (ba, bb):
                        for q in bits(s):
                            for p in bits(s):
                                D2[p, p, q, q] += v
                                D2[p, q, p, q] -= v
                    for q in bits(bb):
                        for p in bits(ba):
                            D2[p, p, q, q] += v
                            D2[q, q, p, p] += v
    return D1, D2


@pytest.mark.parametrize("nbits,n,na,nb,frac", [(64, 6, 3, 2, 1.0),
                                                (128, 6, 3, 3, 0.4),
                                                (256, 5, 1, 3, 0.9)])
def test_rdms_match_pair_sums(nbits, n, na, nb, frac):
    """Against the pair sums in plain Python: a full space, selected lists, a
    zero determinant, a duplicate, a pair below 1e-16 and determinants of
    another electron count. Every element is a sum of at most a few thousand
    terms below 1: 1e-12."""
    T, V, d = fci(n, na, nb, nbits, seed=1)
    d = shuffled(d, seed=5, frac=frac).copy()
    d[3] = 0
    d[7] = d[8]
    d[10:12] = fci(n, na + 1, nb, nbits, seed=1)[2][:2]
    C = np.random.default_rng(2).standard_normal(len(d))
    C /= np.linalg.norm(C)
    C[5] = 1e-17
    H = mb.HamiltonianGenerator(T, V, nbits)
    for two in (True, False):
        o, t = H.form_rdms(d, C, two=two)
        ro, rt = _rdms_by_pairs(d, C, n, two)
        np.testing.assert_allclose(o, ro, rtol=0, atol=1e-12)
        if two:
            np.testing.assert_allclose(t, rt, rtol=0, atol=1e-12)


@pytest.mark.parametrize("n,na,nb,ndets", [(3, 1, 2, 9), (5, 2, 2, 100),
                                           (6, 3, 2, 144), (6, 3, 2, 145),
                                           (7, 2, 3, 196), (7, 2, 3, 197)])
def test_rdms_of_short_lists_and_without_scratch(n, na, nb, ndets):
    """Lists at and one above the length up to which the pairs go straight to
    the 2-RDM (4 n^2), and longer ones without the memory for the sums: an
    allocation that fails is an ENOMEM or, for the sums (the last one), that
    path. Against the pair sums in plain Python: 1e-12 as above."""
    from macis_b200 import _lib
    T, V, d = fci(n, na, nb, 64, seed=1)
    d = shuffled(d, seed=5)[:ndets].copy()
    d[3] = 0
    d[5] = d[6]
    C = np.random.default_rng(2).standard_normal(len(d))
    C /= np.linalg.norm(C)
    H = mb.HamiltonianGenerator(T, V, 64)
    ro, rt = _rdms_by_pairs(d, C, n, True)
    good = 0
    try:
        for k in range(200):
            _lib.check(_lib.LIB.macis_b200_inject_fault(_lib.FAULT_ALLOC, k))
            try:
                o, t = H.form_rdms(d, C)
            except mb.MacisError as e:
                assert e.code == _lib.ENOMEM and good == 0
                continue
            np.testing.assert_allclose(o, ro, rtol=0, atol=1e-12)
            np.testing.assert_allclose(t, rt, rtol=0, atol=1e-12)
            good += 1
            if good == 2:      # without the sums, and with everything
                break
    finally:
        _lib.check(_lib.LIB.macis_b200_inject_fault(_lib.FAULT_NONE, 0))
    assert good == 2


def test_rdm_scratch_of_a_short_list():
    """Ten determinants of 64 orbitals need no multiple of their 2-RDM (134
    MB) beside it: a tenth of it for the tables and what the pool rounds up."""
    from test_gpu_hbuild import _peak_pool_bytes
    n, k = 64, 4
    T, V = mb.synthetic_integrals(n, 1)
    hf = (1 << k) - 1
    a = [hf] + [hf ^ 1 ^ (1 << v) for v in range(k, k + 9)]
    d = mb.sd.make_dets(a, [hf] * 10, 128)
    H = mb.HamiltonianGenerator(T, V, 128)
    C = np.full(10, 10 ** -0.5)
    H.form_rdms(d, C)
    assert _peak_pool_bytes(lambda: H.form_rdms(d, C)) < 1.1 * 8 * n ** 4


@pytest.mark.parametrize("n,ndets", [(16, 130), (17, 40), (17, 1200),
                                     (33, 257)])
def test_rdms_with_more_orbital_pairs_than_threads(n, ndets):
    """Orbital pairs beyond one block's threads and rows beyond one block's,
    straight to the 2-RDM and through the sums (17 orbitals, 1,200
    determinants), against the pair sums in plain Python: 1e-12."""
    rng = np.random.default_rng(n)
    T, V = mb.synthetic_integrals(n, 2)
    hf, words = 7, set()
    while len(words) < ndets:
        a, b = hf, hf
        for _ in range(int(rng.integers(0, 3))):
            i, v = rng.integers(0, 3), rng.integers(3, n)
            x = (1 << int(i)) | (1 << int(v))
            if rng.random() < 0.5:
                a = a ^ x if a & x == 1 << int(i) else a
            else:
                b = b ^ x if b & x == 1 << int(i) else b
        words.add((a, b))
    words = sorted(words)
    d = mb.sd.make_dets([a for a, _ in words], [b for _, b in words], 128)
    d = shuffled(d, seed=1).copy()
    C = rng.standard_normal(len(d))
    C /= np.linalg.norm(C)
    H = mb.HamiltonianGenerator(T, V, 128)
    for two in (True, False):
        o, t = H.form_rdms(d, C, two=two)
        ro, rt = _rdms_by_pairs(d, C, n, two)
        np.testing.assert_allclose(o, ro, rtol=0, atol=1e-12)
        if two:
            np.testing.assert_allclose(t, rt, rtol=0, atol=1e-12)
