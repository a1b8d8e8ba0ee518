"""The FP64 calls' workspace where device memory is short: the queries' minimum is
what the calls took before they had tensor-core scratch, and the pool falls back to
it.  No GPU needed: size queries and a pool that stands in for the allocator."""
import pytest

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def lib():
    from pynof_gb300 import _lib, build

    build.build()
    _lib.load()
    return _lib


def _blocks(*counts):
    return sum((8 * c + 255) // 256 * 256 for c in counts)


def _cases():
    N, P, Q, R = 120, 60, 480, 50
    return {
        "gb_jkj_full_workspace_f64": ((N, P), _blocks(P * N * N)),
        "gb_jkh_mo_full_workspace_f64": ((N, P), _blocks(*[P * N * N] * 3, N * P)),
        "gb_mo_full_workspace_f64": ((N, P), _blocks(N**3 * P, N * N * P * P, N * P)),
        "gb_lagrange2_full_workspace_f64": ((N, P), _blocks(N**3 * P, N * N * P * P, N * P, N * P**3)),
        "gb_mo4_full_workspace_f64": ((N, P, R, P), _blocks(N**3 * P, N * N * R * P)),
        "gb_fock_rc_workspace_f64": ((N, P), _blocks(P * P, P * P)),
        "gb_fock_ro_workspace_f64": ((N, P), _blocks(P * P, P * P, P)),
        "gb_mo_ri_workspace_f64": ((N, P, Q), _blocks(P * N * Q, N * P)),
        "gb_lagrange2_ri_workspace_f64": ((N, P, Q), None),
        "gb_rotate_orbital_workspace_f64": ((500,), _blocks(*[500 * 500] * 6, 1)),
    }


@pytest.mark.parametrize("query", sorted(_cases()))
def test_minimum_leaves_the_scratch_out(lib, query):
    sizes, least = _cases()[query]
    full, low = lib.query(query, *sizes), lib.query_minimum(query, *sizes)
    assert low < full == lib.query(query, *sizes)
    if least is not None:
        assert least - 6 * 256 <= low <= least


@pytest.mark.parametrize("room", ["full", "minimum", "less"])
def test_pool_falls_back_to_the_minimum(lib, monkeypatch, room):
    from pynof_gb300 import ops

    query, (N, P) = "gb_jkj_full_workspace_f64", (60, 30)
    full, low = lib.query(query, N, P), lib.query_minimum(query, N, P)
    limit = {"full": full, "minimum": full - 1, "less": low - 1}[room]

    class Pool:
        def get(self, nbytes, device):
            if nbytes > limit:
                raise torch.OutOfMemoryError("no room")
            return torch.empty(nbytes, dtype=torch.uint8)

    monkeypatch.setattr(ops, "POOL", Pool())
    if room == "less":
        with pytest.raises(torch.OutOfMemoryError):
            ops._ws(query, N, P, device=None)
    else:
        assert ops._ws(query, N, P, device=None)[1] == (full if room == "full" else low)
    # a split-product call has no smaller form
    monkeypatch.setattr(Pool, "get", lambda self, nbytes, device: (_ for _ in ()).throw(torch.OutOfMemoryError()))
    with pytest.raises(torch.OutOfMemoryError):
        ops._ws("gb_jkj_ri_workspace_mixed", 24, 12, 100, 6, device=None)


def test_reservation_is_what_a_solve_needs(lib):
    """A served FP64 solve is admitted by what it cannot do without."""
    from pynof_gb300 import serve, synthetic

    st = synthetic.Structure.for_nbf(300)
    N, Q, P = st.nbf, st.nbfaux, st.nbf5
    held = serve.reservation_bytes(st, "fp64", 6)
    assert held < 8 * (N * N * Q + 2 * N * P * Q + 2 * P * Q + 8 * N * N + 8 * P * P) + 4096
