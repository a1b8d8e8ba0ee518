"""FP64 GEMMs on the tensor cores (seven nine-bit digit planes), through the entry
points that take them above a size: the four-index J and K (packed pairs, K
splits), the generalized Fock matrices (accumulation into the output), the
orbital rotation (products of one matrix with itself) and the FP64 Lagrangian
(batches, a long K).

Tolerances, on the largest element: a sum of K products is exact but for the
dropped digits (2^-53 of the row bounds and less) and one rounding per 1024 k,
and the NumPy float64 reference rounds K times, relative to sums of |a b| that
are at most ~sqrt(K) times the largest result for these operands: 4 sqrt(K) 2^-53
covers both for one GEMM, and three chained ones (K <= 21000) stay below
3 * 4 * 145 * 2^-53 = 2e-13.
"""
import numpy as np
import pytest

from conftest import nrel
from oracle import pynof_oracle as orc

pytestmark = pytest.mark.gpu
TOL = 2e-13


@pytest.fixture(scope="module")
def ops():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from pynof_gb300 import ops as o

    return o


def _host(*ts):
    return [t.cpu().numpy() for t in ts]


def _eri(N, rng):
    f = rng.standard_normal((N, N, N)) * np.exp(-0.05 * (np.arange(N)[:, None] + np.arange(N)[None, :]))[:, :, None]
    f = (0.5 * (f + f.transpose(1, 0, 2))).reshape(N * N, N)
    return (f @ f.T).reshape(N, N, N, N)


@pytest.mark.parametrize("N,P", [(40, 20), (53, 33), (64, 64), (67, 13)])
def test_four_index_jk(ops, N, P):
    rng = np.random.default_rng(N)
    I, C = _eri(N, rng), np.linalg.qr(rng.standard_normal((N, N)))[0]
    J, K = _host(*ops.jkj_full(ops.to_device(C), ops.to_device(I), P))
    D = np.einsum("si,li->isl", C[:, :P], C[:, :P])
    assert nrel(J, np.einsum("isl,mnsl->imn", D, I, optimize=True)) < TOL
    assert nrel(K, np.einsum("inl,mnsl->ims", D, I, optimize=True)) < TOL


@pytest.mark.parametrize("N,P,nbeta", [(131, 70, 14), (97, 97, 20), (160, 40, 8)])
def test_fock_accumulates(ops, N, P, nbeta):
    rng = np.random.default_rng(N + P)
    J, K = rng.standard_normal((2, P, N, N))
    n, H = rng.random(P), rng.standard_normal((N, N))
    cj, ck = rng.standard_normal((2, P, P))
    np.fill_diagonal(cj, 0.0)
    np.fill_diagonal(ck, 0.0)
    F, = _host(ops.fock_rc(*(ops.to_device(x) for x in (J, K, n, H, cj, ck)), nbeta, nbeta))
    ref = n[:, None, None] * (H + J) + np.einsum("ij,jmn->imn", cj, J) - np.einsum("ij,jmn->imn", ck, K)
    assert nrel(F, ref) < TOL


@pytest.mark.parametrize("N,P", [(300, 150), (333, 41), (512, 256)])
def test_rotation_of_large_orbitals(ops, N, P):
    from scipy.linalg import expm

    rng = np.random.default_rng(N)
    C = np.linalg.qr(rng.standard_normal((N, N)))[0]
    i, j = np.triu_indices(N, 1)
    keep = i < P
    y = 0.05 * rng.standard_normal(keep.sum())
    Y = np.zeros((N, N))
    Y[i[keep], j[keep]] = y
    got, = _host(ops.rotate_orbital(ops.to_device(y), ops.to_device(C), P))
    assert nrel(got, C @ expm(Y - Y.T)) < TOL


@pytest.mark.parametrize("nbf,naux,nbf5", [(97, 305, 40), (128, 512, 64), (65, 257, 65)])
def test_lagrangian(ops, nbf, naux, nbf5):
    from pynof_gb300 import synthetic

    st = synthetic.Structure(nbf=nbf, nbfaux=naux, ndoc=1, ncwo=nbf5 - 1)
    b, C, H, n = synthetic.make_inputs(st, nbf)
    cj, ck = 2 * np.outer(n, n), np.outer(n, n)
    got, hmat = _host(*ops.lagrange2_ri(*(ops.to_device(x) for x in (C, H, b, n, cj, ck)), nbf5, st.nbeta, st.nalpha))
    ref, href = orc.lagrange2(n, cj.copy(), ck.copy(), C, H, None, b, st)
    assert nrel(got, ref) < TOL and nrel(hmat, href) < TOL


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_nonfinite_operands_take_fp64_arithmetic(ops, bad):
    """A NaN or an infinity goes through the products as FP64 arithmetic has it,
    leaves the status word clear, and does not touch a call that follows."""
    N, P = 53, 33
    rng = np.random.default_rng(3)
    I, C = _eri(N, rng), np.linalg.qr(rng.standard_normal((N, N)))[0]
    good = _host(*ops.jkj_full(ops.to_device(C), ops.to_device(I), P))
    C2 = C.copy()
    C2[5, 4] = bad  # orbital 4 alone
    J, K = _host(*ops.jkj_full(ops.to_device(C2), ops.to_device(I), P))
    ops.check_device_status()
    others = [i for i in range(P) if i != 4]
    for got, ref in ((J, good[0]), (K, good[1])):
        assert not np.isfinite(got[4]).any()
        assert nrel(got[others], ref[others]) < TOL
    again = _host(*ops.jkj_full(ops.to_device(C), ops.to_device(I), P))
    assert all(np.array_equal(x, y) for x, y in zip(again, good))


def _product(ops, A, B):
    """A B for A (K, K) without a diagonal and B (K, N^2) through fock_rc, whose
    other terms are zero here (n = 0, H = 0, ck12 = 0)."""
    K, N = A.shape[0], int(round(B.shape[1] ** 0.5))
    J, z = ops.to_device(B.reshape(K, N, N)), ops.to_device(np.zeros((K, K)))
    F = ops.fock_rc(J, J, ops.to_device(np.zeros(K)), ops.to_device(np.zeros((N, N))), ops.to_device(A), z, 1, 1)
    return F.cpu().numpy().reshape(K, N * N)


def _element_error(got, A, B, rows=slice(None), cols=slice(None)):
    """Largest |got - A B| over sum_k |a_k b_k|, in units of 2^-53, in extended precision."""
    a, b = A[rows].astype(np.longdouble), B[:, cols].astype(np.longdouble)
    ref = np.zeros((a.shape[0], b.shape[1]), dtype=np.longdouble)
    size = ref.copy()
    for k in range(a.shape[1]):
        t = a[:, k, None] * b[None, k]
        ref += t
        size += np.abs(t)
    err = np.abs(got[rows][:, cols] - ref)
    assert (err[size == 0] == 0).all()
    return float((err[size > 0] / size[size > 0]).max() * 2.0**53)


# An FP64 sum of K products is off by at most K 2^-53 sum |a b|, and by ~sqrt(K) of it
# where the roundings are independent: 2 sqrt(K) for every element holds a product to
# what FP64 arithmetic gives element by element (a lost bit per factor of two beyond).
@pytest.mark.parametrize("spread", [0, 10, 20, 40, 200])
@pytest.mark.parametrize("P,N", [(40, 230), (150, 150)])
def test_graded_operands_keep_fp64_accuracy(ops, P, N, spread):
    """Columns of A scaled by d_k and rows of B by 1 / d_k, d_k over 2^spread: every
    element's leading terms are far below the product of its row bounds."""
    rng = np.random.default_rng(P + spread)
    A, B = rng.standard_normal((P, P)), rng.standard_normal((P, N * N))
    np.fill_diagonal(A, 0.0)
    d = np.exp2(np.rint(spread * rng.random(P)))
    assert _element_error(_product(ops, A * d, B / d[:, None]), A * d, B / d[:, None], cols=slice(0, N * N, 37)) < \
        2 * np.sqrt(P)


def test_one_graded_row_among_ungraded(ops):
    """Row 77 alone meets one column alone badly; the rest of the output is as it was,
    and products that are all zero give zero."""
    P, N = 150, 150
    rng = np.random.default_rng(5)
    A, B = rng.standard_normal((P, P)), rng.standard_normal((P, N * N))
    np.fill_diagonal(A, 0.0)
    plain = _product(ops, A, B)
    A[77, 0], B[0, 5000] = 1e9, 1e-9  # the row's bound is in k = 0, the column has nothing there
    A[3], B[:, 200] = 0.0, 0.0
    A[3, ::2], B[1::2, 200] = 1.0, 1.0
    A[3, 3] = 0.0
    got = _product(ops, A, B)
    assert _element_error(got, A, B, rows=[3, 77, 78], cols=slice(4900, 5100)) < 2 * np.sqrt(P)
    assert _element_error(got, A, B, rows=slice(0, P, 9), cols=slice(0, N * N, 101)) < 2 * np.sqrt(P)
    assert got[3, 200] == 0.0
    keep = np.ones_like(got, dtype=bool)
    keep[[3, 77]], keep[:, [200, 5000]] = False, False
    assert nrel(got[keep], (A @ B)[keep]) < TOL and nrel(plain[keep], got[keep]) < 1e-8


@pytest.mark.parametrize("spread", [0, 20, 60])
def test_graded_k_splits(ops, spread):
    """The same through a long K in splits and packed output pairs (J of the four-index
    route; D is rounded once more on the way)."""
    N, P = 60, 40
    rng = np.random.default_rng(spread)
    I, C = rng.standard_normal((N, N, N, N)), rng.standard_normal((N, N))
    I = I + I.transpose(1, 0, 2, 3)
    d = np.exp2(np.rint(0.5 * spread * rng.random(N)))
    C, I = C * d[:, None], I / d[:, None] / d
    J, _ = ops.jkj_full(ops.to_device(C), ops.to_device(I), P)
    D = np.einsum("si,li->isl", C[:, :P], C[:, :P]).reshape(P, N * N)
    assert _element_error(J.cpu().numpy().reshape(P, N * N), D, I.reshape(N * N, N * N).T,
                          rows=slice(0, P, 7), cols=slice(0, N * N, 61)) < 2 * N + 1


@pytest.fixture
def small_panels(ops):
    """2 MB of slices at a time: what takes several GB of them otherwise runs in panels."""
    from pynof_gb300 import _lib

    _lib.call("gb_test_panel_bytes", 2 << 20)
    yield
    _lib.call("gb_test_panel_bytes", 0)


@pytest.mark.parametrize("N,P", [(64, 60), (66, 66), (53, 33)])
def test_panels_of_packed_pairs(ops, small_panels, N, P):
    """Row panels on either side (the pairs are the tiles' rows at P = 60, their columns
    at P = 66) with K splits, graded rows in one panel, and a NaN in the last one only."""
    rng = np.random.default_rng(N)
    I, C = _eri(N, rng), np.linalg.qr(rng.standard_normal((N, N)))[0]
    D = np.einsum("si,li->isl", C[:, :P], C[:, :P])
    Jr, Kr = np.einsum("isl,mnsl->imn", D, I, optimize=True), np.einsum("inl,mnsl->ims", D, I, optimize=True)
    J, K = _host(*ops.jkj_full(ops.to_device(C), ops.to_device(I), P))
    assert nrel(J, Jr) < TOL and nrel(K, Kr) < TOL
    m = N - 1
    I2 = I.copy()
    I2[m, m, 0, 0] = np.nan  # the last pair of J; K of row m and column 0
    J, _ = _host(*ops.jkj_full(ops.to_device(C), ops.to_device(I2), P))
    assert np.isnan(J[:, m, m]).all()
    J[:, m, m] = Jr[:, m, m]
    assert nrel(J, Jr) < TOL
    I3 = I.copy()
    I3[m, m] = 1e-12 * rng.standard_normal((N, N))
    I3[m, m, 0, 0] = 1.0 / max(abs(D[0, 0, 0]), 1e-3)
    C3 = C.copy()
    C3[0] *= 1e-10  # what meets the bound of pair (m, m) is far below it
    J, _ = _host(*ops.jkj_full(ops.to_device(C3), ops.to_device(I3), P))
    D3 = np.einsum("si,li->isl", C3[:, :P], C3[:, :P]).reshape(P, N * N)
    assert _element_error(J.reshape(P, N * N), D3, I3.reshape(N * N, N * N).T, rows=slice(0, P, 5),
                          cols=[0, N + 1, m * N, m * N + m]) < 2 * N + 1


def test_panels_of_a_batch_and_in_place(ops, small_panels):
    """Batch panels with one shared operand and a ragged last one (the MO transforms),
    row panels of a GEMM that adds to its output (the Fock matrices)."""
    test_lagrangian(ops, 97, 305, 40)
    test_fock_accumulates(ops, 131, 70, 14)
    test_graded_operands_keep_fp64_accuracy(ops, 40, 230, 20)


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_panels_with_nonfinite_operands(ops, small_panels, bad):
    test_nonfinite_operands_take_fp64_arithmetic(ops, bad)


def test_without_scratch(ops, monkeypatch):
    """Where the pool has no room for the scratch, the calls run on what they needed
    before (on the FP64 units)."""
    from pynof_gb300 import _lib

    torch = pytest.importorskip("torch")
    N, P = 53, 33
    rng = np.random.default_rng(N)
    I, C = _eri(N, rng), np.linalg.qr(rng.standard_normal((N, N)))[0]
    real, least = ops.WorkspacePool(), _lib.query_minimum("gb_jkj_full_workspace_f64", N, P)

    class Pool:
        def get(self, nbytes, device):
            if nbytes > least:
                raise torch.OutOfMemoryError("no room")
            return real.get(nbytes, device)

    monkeypatch.setattr(ops, "POOL", Pool())
    J, K = _host(*ops.jkj_full(ops.to_device(C), ops.to_device(I), P))
    D = np.einsum("si,li->isl", C[:, :P], C[:, :P])
    assert nrel(J, np.einsum("isl,mnsl->imn", D, I, optimize=True)) < TOL
    assert nrel(K, np.einsum("inl,mnsl->ims", D, I, optimize=True)) < TOL


@pytest.mark.parametrize("N", [24, 29, 31, 36, 43])
def test_sizes_where_the_rule_changes_units(ops, N):
    """Small sizes on both sides of the line between the FP64 units and the tensor cores,
    through every kind of GEMM that takes them."""
    P, Q = N // 2, 3 * N + 5
    test_four_index_jk(ops, N, P)
    test_lagrangian(ops, N, Q, P)
    test_fock_accumulates(ops, 4 * N, P, max(1, P // 5))
    rng = np.random.default_rng(N)
    I, C, H = _eri(N, rng), np.linalg.qr(rng.standard_normal((N, N)))[0], rng.standard_normal((N, N))
    dC, dI = ops.to_device(C), ops.to_device(I)
    hm, imo = _host(*ops.mo_full(dC, ops.to_device(H), dI, P))
    Cp = C[:, :P]
    ref = np.einsum("mp,nq,mnsl,sr,lt->pqrt", C, Cp, I, Cp, Cp, optimize=True)
    assert nrel(imo, ref) < TOL and nrel(hm, C.T @ H @ Cp) < TOL
    m4, = _host(ops.mo4_full(dC, dI, (1, P), (0, N), (2, N), (0, P)))
    assert nrel(m4, np.einsum("mp,nq,mnsl,sr,lt->pqrt", C[:, 1:P], C, I, C[:, 2:], Cp, optimize=True)) < TOL


@pytest.mark.parametrize("spread", [0, 40])
def test_graded_rows_in_place(ops, spread):
    """F = cj J - ck K adds to its output in place: tiles left to FP64 arithmetic beside
    tiles that are stored, each added once."""
    P, N = 150, 150
    rng = np.random.default_rng(spread)
    J, K = rng.standard_normal((2, P, N * N))
    cj, ck = rng.standard_normal((2, P, P))
    np.fill_diagonal(cj, 0.0)
    np.fill_diagonal(ck, 0.0)
    ck[[5, 149], 0], K[0, [70, 10000]] = 2.0**spread, 2.0**-spread
    z = ops.to_device(np.zeros(P))
    F, = _host(ops.fock_rc(*(ops.to_device(x.reshape(P, N, N)) for x in (J, K)), z, ops.to_device(np.zeros((N, N))),
                           ops.to_device(cj), ops.to_device(ck), 1, 1))
    F, ref = F.reshape(P, N * N), cj @ J - ck @ K
    rows = np.setdiff1d(np.arange(P), [5, 149])
    assert nrel(F[rows], ref[rows]) < TOL
    assert _element_error(-F, np.concatenate([-cj, ck], 1), np.concatenate([J, K], 0), rows=[5, 6, 149],
                          cols=[0, 70, 71, 9999, 10000]) < 2 * np.sqrt(2 * P)
