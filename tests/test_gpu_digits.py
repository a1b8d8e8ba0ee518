"""Nine-bit digit slices (split code 6): chunks, carries and tile edges.

The leading digit groups are exact sums in FP32 chunks whose length the kernel
takes from the digits' norms.  Operands whose digits are all as large as they
get (equal rows, one sign) make every chunk as full as it can be: a chunk too
long, or a carry lost between groups, would show as an error of 2^-24 and more.

Tolerance, relative to the largest |C| (which is K 2^(Ea + Eb) up to a factor of
4 for these operands): the dropped products s + t > 6 are at most
4 * 2^16 * 2^-61 * 1.01 < 2^-42.9 per k, the slicing error 2 * 2^-45, and the FP32
group, at most 2^-25 per k, loses at most 2^-24 of itself in each of its
9 K / 16 additions: 2^-49.8 K.  For K <= 1300 that is below
4 (2^-42.9 + 2^-44 + 2^-39.4) < 2^-37 = 7.3e-12.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = 2.0 ** -37


@pytest.fixture(scope="module")
def ops():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from pynof_gb300 import ops as o

    return o


def _operands(kind, M, N, K):
    rng = np.random.default_rng(M + 3 * N + 7 * K)
    if kind == "full":  # every digit 255 or 256 of one sign: x just below 1
        x = 1.0 - 2.0 ** -40 * rng.integers(1, 3, K)
        return np.tile(x, (M, 1)), np.tile(x, (N, 1))
    if kind == "halves":  # balanced digits at their bound: +-256 in every place
        x = sum(256.0 * 2.0 ** -(9 * s - 1) * (1 if s == 1 else 0.5) for s in range(1, 6)) * 0.5
        sg = np.where(rng.random(K) < 0.5, -1.0, 1.0)
        return np.tile(x * sg, (M, 1)), np.tile(x * sg, (N, 1))
    a = rng.standard_normal((max(M, N), K))  # equal rows of A and B: sums of squares
    return a[:M].copy(), a[:N].copy()


@pytest.mark.parametrize("kind", ["full", "halves", "gauss"])
@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (128, 128, 47), (129, 127, 48), (130, 104, 49), (127, 105, 128),
                                   (200, 260, 129), (64, 300, 257), (257, 48, 400), (128, 176, 1300)])
def test_full_chunks_and_tile_edges(ops, kind, M, N, K):
    A, B = _operands(kind, M, N, K)
    ref = A @ B.T
    C = ops.dgemm_mixed(ops.to_device(A), ops.to_device(B), 6).cpu().numpy()
    ops.check_device_status()
    err = np.max(np.abs(C - ref)) / np.max(np.abs(ref))
    assert err < TOL, err


@pytest.mark.parametrize("nbf,naux,nbf5", [(3, 5, 2), (24, 116, 24), (70, 129, 33), (150, 500, 70)])
def test_build_with_equal_orbitals(ops, nbf, naux, nbf5):
    """The JK build (persistent kernel, symmetric tiles) on a factor and
    orbitals of one sign and nearly one size, against float64."""
    rng = np.random.default_rng(nbf)
    b = 1.0 - 2.0 ** -30 * rng.random((nbf, nbf, naux))
    b = 0.5 * (b + b.transpose(1, 0, 2))
    C = 1.0 - 2.0 ** -30 * rng.random((nbf, nbf))
    T = np.einsum("mq,mnl->qnl", C[:, :nbf5], b)
    d = np.einsum("nq,qnl->ql", C[:, :nbf5], T)
    J, K = np.einsum("ql,mnl->qmn", d, b), np.einsum("qml,qnl->qmn", T, T)
    dJ, dK = ops.jkj_ri_mixed(ops.to_device(C), ops.PreparedRI(ops.to_device(b), 6), nbf5)
    ops.check_device_status()
    for got, ref in ((dJ, J), (dK, K)):
        assert np.max(np.abs(got.cpu().numpy() - ref)) / np.max(np.abs(ref)) < 3 * TOL


@pytest.mark.parametrize("nbf,naux,nbf5", [(20, 41, 1), (40, 70, 17), (150, 130, 128), (140, 90, 129), (210, 60, 207)])
def test_symmetric_mo_transform(ops, nbf, naux, nbf5):
    """(pq|l) computed for q <= p: J_MO, K_MO and the Lagrangian around the edges
    of the 128- and 16-column steps, against the FP64 path.  The split's error
    is a few 2^-45 of the row bounds per k (TOL above); K_MO and the Lagrangian
    square or contract (pq|l), which doubles it."""
    rng = np.random.default_rng(nbf5)
    b = rng.standard_normal((nbf, nbf, naux))
    b = ops.to_device(0.5 * (b + b.transpose(1, 0, 2)))
    C = ops.to_device(np.linalg.qr(rng.standard_normal((nbf, nbf)))[0])
    H = rng.standard_normal((nbf, nbf))
    H, n = ops.to_device(H + H.T), rng.random(nbf5)
    cj, ck = ops.to_device(2 * np.outer(n, n)), ops.to_device(np.outer(n, n))
    n, prep = ops.to_device(n), ops.PreparedRI(b, 6)
    ref = ops.jkh_mo_ri(C, H, b, nbf5) + ops.lagrange2_ri(C, H, b, n, cj, ck, nbf5, 1, 1)
    got = ops.jkh_lagrange2_ri_mixed(C, H, prep, n, cj, ck, nbf5, 1, 1)
    mo = ops.jkh_mo_ri_mixed(C, H, prep, nbf5)
    ops.check_device_status()
    for x, r in zip(got + mo, ref + ref[:3]):
        x, r = x.cpu().numpy(), r.cpu().numpy()
        assert np.max(np.abs(x - r)) / np.max(np.abs(r)) < 4 * TOL


def _all_255(places):
    """The number below 1 whose nine-bit digits are all 255."""
    return sum(255 * 2.0 ** -(9 * s - 1) for s in range(1, places + 1))


@pytest.mark.parametrize("K", [4095, 4096, 4097, 6100])
def test_full_digits_over_a_long_k(ops, K):
    """Both drains at their longest: 32-bit pairs up to K = 4096, 64-bit sums and the FP32
    group per chunk beyond.  The bound of TOL above at this K: 4 (2^-42.9 + 2^-44 +
    2^-49.8 K)."""
    tol = 4 * (2.0**-42.9 + 2.0**-44 + 2.0**-49.8 * K)
    x = _all_255(5)
    M, N = 130, 104
    sg = np.where(np.random.default_rng(K).random(K) < 0.5, -x, x)
    for a, b in ((np.full(K, x), np.full(K, x)), (sg, sg)):
        C = ops.dgemm_mixed(ops.to_device(np.tile(a, (M, 1))), ops.to_device(np.tile(b, (N, 1))), 6).cpu().numpy()
        assert np.max(np.abs(C / (K * x * x) - 1.0)) < tol
    # the persistent kernel: J of a factor and orbitals of that size (K = naux)
    nbf = 20
    db = ops.to_device(np.full((nbf, nbf, K), x))
    J, Km = ops.jkj_ri_mixed(ops.to_device(np.full((nbf, nbf), x)), ops.PreparedRI(db, 6), 3)
    ops.check_device_status()
    T = nbf * x * x
    assert np.max(np.abs(J.cpu().numpy() / (K * nbf * x * T * x) - 1.0)) < 3 * tol
    assert np.max(np.abs(Km.cpu().numpy() / (K * T * T) - 1.0)) < 3 * tol


def test_full_digits_of_the_fp64_engine(ops):
    """Six planes of 255 (53 bits) in both operands, K past the 1024 of one integer sum,
    through the Fock matrices' product (n = 0, H = 0, ck12 = 0).  The sum is exact but for
    two roundings to FP64 and, relative to it, the dropped digit products (6 * 2^-63) and
    the FP32 group's own roundings (2^-57): 2^-52."""
    torch = pytest.importorskip("torch")
    from fractions import Fraction

    P, x = 1030, _all_255(6)
    exact = float((P - 1) * Fraction(x) ** 2)
    J = torch.full((P, P, P), x, dtype=torch.float64, device="cuda")
    cj = torch.full((P, P), x, dtype=torch.float64, device="cuda")
    z = torch.zeros((P, P), dtype=torch.float64, device="cuda")
    F = ops.fock_rc(J, J, z[0].contiguous(), z, cj, z, 1, 1)
    assert float((F / exact - 1.0).abs().max()) <= 2.0**-52
    sg = torch.where(torch.arange(P, device="cuda") % 3 == 0, -1.0, 1.0).double()
    F = ops.fock_rc(J * sg[:, None, None], J, z[0].contiguous(), z, cj * sg[None, :], z, 1, 1)
    assert float((F / exact - 1.0).abs().max()) <= 2.0**-52
