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
