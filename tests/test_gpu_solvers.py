"""SpMV and Davidson on the GPU against the reference and the golden
energies (davidson.cxx:48, tolerance 1e-8 Eh), FP64 and mixed precision."""
import numpy as np
import pytest

import macis_b200 as mb
from cases import fci, shuffled
from golden_data import constants, water

pytestmark = pytest.mark.gpu
K = constants()


@pytest.fixture(scope="module")
def water_cisd(port):
    norb, T, V, ec = water()
    dets = port.cisd_space(64, norb, 5, 5)
    H = mb.HamiltonianGenerator(T, V, 64, norb)
    return norb, T, V, ec, dets, H


def test_spmv_matches_reference(ref, water_cisd):
    norb, T, V, _, dets, H = water_cisd
    A = mb.make_csr_hamiltonian(dets, H, 1e-16)
    R = ref.csr(ref.ham(64, norb, T, V), dets, dets, 1e-16)
    rng = np.random.default_rng(0)
    for _ in range(3):
        x = rng.standard_normal(A.n)
        y = A.spmv(x)
        yr = R.spmv(x)
        np.testing.assert_allclose(y, yr, rtol=1e-12, atol=1e-12 * np.abs(yr).max())
    # alpha / beta and block of K = 3 columns
    X = rng.standard_normal((3, A.n))
    Y0 = rng.standard_normal((3, A.m))
    Y = Y0.copy()
    from macis_b200._lib import LIB, check
    check(LIB.macis_b200_spmv(A.handle, 3, 0.5, X.ctypes.data, A.n, -2.0,
                              Y.ctypes.data, A.m, 0))
    for k in range(3):
        np.testing.assert_allclose(Y[k], 0.5 * R.spmv(X[k]) - 2.0 * Y0[k],
                                   rtol=1e-11, atol=1e-10)


def test_davidson_water_golden(water_cisd):
    norb, T, V, ec, dets, H = water_cisd
    A = mb.make_csr_hamiltonian(dets, H, 1e-16)
    X = np.zeros(A.n)
    mb.diagonal_guess(A.n, A, X)
    it, E = mb.davidson(A.n, 15, mb.SparseMatrixOperator(A), A.diagonal(),
                        1e-8, X)
    assert abs(E + ec - K["water_cisd_e0_plus_ecore"]) < 1e-8
    assert abs(np.linalg.norm(X) - 1.0) < 1e-10
    assert abs(X @ A.spmv(X) - E) < 1e-8


def test_davidson_vs_reference_c1(ref):
    # The synthetic integrals are strongly correlated: the reference solver
    # (no restart) needs ~190 basis vectors at 1e-8, so both sides get 300.
    T, V, dets = fci(10, 5, 5, 64, seed=0)
    H = mb.HamiltonianGenerator(T, V, 64)
    E, X = mb.selected_ci_diag(dets, H, np.finfo(float).eps, 300, 1e-8)
    Er, Xr = ref.selected_ci_diag(ref.ham(64, 10, T, V), dets,
                                  np.finfo(float).eps, 300, 1e-8)
    assert abs(E - Er) < 1e-8
    assert abs(abs(X @ Xr) - 1.0) < 1e-7
    # thick restart reaches the same root with a 40-vector basis
    E2, X2 = mb.selected_ci_diag(dets, H, np.finfo(float).eps, 40, 1e-8,
                                 restart_keep=8, max_iter=2000)
    assert abs(E2 - Er) < 1e-8
    with pytest.raises(RuntimeError, match="Davidson Did Not Converge!"):
        mb.selected_ci_diag(dets, H, np.finfo(float).eps, 20, 1e-8)


def test_mixed_precision_energy():
    T, V, dets = fci(10, 5, 5, 64, seed=0)
    H = mb.HamiltonianGenerator(T, V, 64)
    kw = dict(restart_keep=8, max_iter=2000)
    E64, _ = mb.selected_ci_diag(dets, H, np.finfo(float).eps, 40, 1e-8, **kw)
    E32, X = mb.selected_ci_diag(dets, H, np.finfo(float).eps, 40, 1e-8,
                                 precision=mb.MIXED, **kw)
    assert abs(E32 - E64) < 1e-7          # north-star mixed target
    assert abs(np.linalg.norm(X) - 1.0) < 1e-10


def test_davidson_nonconvergence_raises():
    T, V, dets = fci(8, 4, 4, 64, seed=1)
    H = mb.HamiltonianGenerator(T, V, 64)
    A = mb.make_csr_hamiltonian(dets, H, 1e-14)
    X = np.zeros(A.n)
    with pytest.raises(RuntimeError, match="Davidson Did Not Converge!"):
        mb.davidson(A.n, 3, mb.SparseMatrixOperator(A), None, 1e-14, X,
                    use_guess=False)


def test_guess_reuse_and_selected_space(ref):
    T, V, dets = fci(9, 4, 4, 128, seed=4)
    sel = shuffled(dets, seed=5, frac=0.5)
    H = mb.HamiltonianGenerator(T, V, 128)
    E, X = mb.selected_ci_diag(sel, H, 1e-12, 300, 1e-9)
    Er, _ = ref.selected_ci_diag(ref.ham(128, 9, T, V), sel, 1e-12, 300, 1e-9)
    assert abs(E - Er) < 1e-8
    E2, X2 = mb.selected_ci_diag(sel, H, 1e-12, 300, 1e-9, C=X)
    assert abs(E2 - E) < 1e-8


@pytest.mark.parametrize("n,na,nb", [(2, 1, 1), (4, 2, 1), (6, 3, 3), (7, 3, 4),
                                     (8, 3, 4)])
@pytest.mark.parametrize("max_m,keep", [(40, 8), (40, 12), (140, 10), (300, 0)])
def test_davidson_against_dense(n, na, nb, max_m, keep):
    """Lowest eigenpair against numpy's of the dense matrix: vectors from a
    few rows to several blocks of rows, Ritz vectors above and below the
    length that travels with the launch (128), restarts keeping more and
    fewer columns than a thread holds. E to 1e-8 (residual 1e-9 over a gap
    above 1e-2 squares to far less), the vector to 1e-6."""
    T, V, d = fci(n, na, nb, 64, seed=3)
    H = mb.HamiltonianGenerator(T, V, 64)
    A = mb.make_csr_hamiltonian(d, H, np.finfo(float).eps)
    rp, ci, nz = A.to_host()
    M = np.zeros((A.m, A.m))
    for i in range(A.m):
        M[i, ci[rp[i]:rp[i + 1]]] = nz[rp[i]:rp[i + 1]]
    w, U = np.linalg.eigh(M)
    X = np.zeros(A.n)
    keep = min(keep, max(min(max_m, A.n) - 1, 0))
    it, E = mb.davidson(A.n, max_m, A, None, 1e-9, X, use_guess=False,
                        restart_keep=keep, max_iter=3000)
    assert abs(E - w[0]) < 1e-8
    if len(w) == 1 or w[1] - w[0] > 1e-2:
        assert abs(abs(U[:, 0] @ X) - 1.0) < 1e-6
    st = mb.davidson_stats()
    assert st["iterations"] == it and all(v >= 0 for v in st.values())


@pytest.mark.parametrize("stored", [True, False])
@pytest.mark.parametrize("n,na,nb,max_m", [(1, 1, 0, 1), (2, 2, 2, 40),
                                           (2, 1, 1, 1), (2, 1, 1, 2),
                                           (6, 3, 3, 1), (6, 3, 3, 2)])
def test_davidson_smallest_subspaces(n, na, nb, max_m, stored):
    """A single determinant (E is its diagonal element, the vector the unit
    vector) and the smallest subspaces, where the solver stops after one step
    with the basis (x0, H x0): the lowest pair of numpy's 2 x 2 projection.
    Entries of order 10 in sums of 400 at most: 1e-9."""
    from macis_b200 import _lib
    T, V, d = fci(n, na, nb, 64, seed=3)
    H = mb.HamiltonianGenerator(T, V, 64)
    A = mb.make_csr_hamiltonian(d, H, 0.0)
    rp, ci, nz = A.to_host()
    M = np.zeros((A.m, A.m))
    for i in range(A.m):
        M[i, ci[rp[i]:rp[i + 1]]] = nz[rp[i]:rp[i + 1]]
    op = A if stored else mb.MatrixFreeHamiltonian(d, H, 0.0)
    solve = (_lib.LIB.macis_b200_davidson_ex if stored
             else _lib.LIB.macis_b200_hop_davidson)
    import ctypes as C
    X, E, it = np.zeros(A.m), C.c_double(), C.c_int64()
    o = _lib.DavidsonOptsC(max_m, 1e-13, 0, 0, 0)
    rc = solve(op.handle, C.byref(o), X.ctypes.data, C.byref(E), C.byref(it), 0)
    assert it.value == 1
    if A.m == 1:
        assert rc == 0 and E.value == M[0, 0] and X[0] == 1.0
        return
    assert rc == _lib.ENOCONV
    Q = np.linalg.qr(np.stack([np.eye(A.m)[np.argmin(np.diag(M))],
                               M[:, np.argmin(np.diag(M))]], axis=1))[0]
    w, U = np.linalg.eigh(Q.T @ M @ Q)
    assert abs(E.value - w[0]) < 1e-9
    assert abs(abs(X @ Q @ U[:, 0]) - 1.0) < 1e-9


@pytest.mark.parametrize("stored", [True, False])
def test_product_time_leaves_host_work_out(stored):
    """The products' device time does not count what the GPU waits for: a
    subspace of 1,000 vectors has the host clear 8 MB of Rayleigh matrix
    between the first step and the first product (4 ms, 0.4 ms at 20 GB/s),
    while a product of 3,136 determinants (1.4e6 elements, 17 MB) takes some
    10 us stored and some 100 us matrix-free."""
    T, V, d = fci(8, 3, 3, 64, seed=2)
    H = mb.HamiltonianGenerator(T, V, 64)
    A = (mb.make_csr_hamiltonian(d, H, 0.0) if stored
         else mb.MatrixFreeHamiltonian(d, H, 0.0))
    for _ in range(2):       # the second time with everything loaded
        with pytest.raises(RuntimeError, match="Did Not Converge"):
            mb.davidson(len(d), 1000, A, None, 1e-14, np.zeros(len(d)),
                        use_guess=False, max_iter=1)
    st = mb.davidson_stats()
    assert st["iterations"] == 1
    assert 0 < st["apply_ms"] < 0.3
    dev = sum(st[k] for k in ("apply_ms", "rayleigh_ms", "residual_ms",
                              "ortho_ms"))
    assert dev < st["wall_ms"]


@pytest.mark.parametrize("rows", [1, 7, 32767, 32768, 32801])
def test_spmv_at_the_block_shapes(rows):
    """Products of row blocks below and above the length from which 32 and not
    8 rows make a block, against numpy on the downloaded matrix: FP64, and
    FP32 values with the FP32 copy of x. Sums of at most 876 terms: 1e-12 of
    the largest."""
    T, V, d = fci(10, 5, 5, 64, seed=0)
    H = mb.HamiltonianGenerator(T, V, 64)
    x = np.random.default_rng(1).standard_normal(len(d))
    for vt in (np.float64, np.float32):
        A = mb.make_csr_hamiltonian_block(d[:rows], d, H, 1e-14, value_t=vt)
        rp, ci, nz = A.to_host()
        xs = x if vt is np.float64 else x.astype(np.float32).astype(np.float64)
        ref = np.add.reduceat(nz.astype(np.float64) * xs[ci], rp[:-1])
        if vt is np.float32:
            ref += A.diagonal() * x[:rows]
        np.testing.assert_allclose(A.spmv(x), ref, rtol=0,
                                   atol=1e-12 * np.abs(ref).max())
