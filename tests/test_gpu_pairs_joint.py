"""Pair kernels over joint sites: energies, counts and weighted bimarginals at
the edges of their tiles, for every tile configuration (q <= 21) and the
first alphabet past them."""
import numpy as np
import pytest

from oracle import oracle
from mi3gpu_b200 import _lib
from tests._util import dev, host, empty, stream, random_model

pytestmark = pytest.mark.gpu

# alphabets at the lines between configurations, lengths around one and two
# blocks of 8, 16 and 32 sites, and sequences around one and several chunks
QS = [1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 20, 21, 22]
LN = [(2, 33), (15, 1024), (16, 1025), (33, 4097), (65, 777)]


@pytest.mark.parametrize("q", QS)
@pytest.mark.parametrize("L,N", LN)
def test_pair_kernels_at_tile_edges(cuda, L, q, N):
    rng = np.random.default_rng(1000 * q + L)
    J = random_model(L, q, 7 * q + L)
    # the buffer is longer than the sequences used
    mem = oracle.pack_seqs(rng.integers(0, q, size=(N + 5, L)).astype("<u1"))
    w = rng.uniform(0.01, 3.0, size=N).astype("<f4")
    np_, qq, B = L * (L - 1) // 2, q * q, N + 5
    dm, dJ, dw = dev(mem), dev(J), dev(w)

    E = empty((N,), np.float32)
    ws = empty((N + 1,), np.int64)
    _lib.call("mi3_energies", dJ.data_ptr(), dm.data_ptr(), B, N, E.data_ptr(), L, q, ws.data_ptr(), ws.numel() * 8,
              stream())
    e64 = oracle.energies_f64(J, mem, L, q)[:N]
    # a coupling is rounded in float 15 times at most (pair-major rows of 16),
    # 4 to 6 times over joint sites: below 2^-20 of the sum of magnitudes; then
    # the final rounding
    mag = oracle.energies_f64(np.abs(J), mem, L, q)[:N]
    assert np.all(np.abs(host(E) - e64) <= 2.0 ** -20 * mag + 2.0 ** -23 * np.abs(e64) + 1e-9)

    cnt = empty((np_, qq), np.uint32)
    _lib.call("mi3_bicounts", dm.data_ptr(), B, N, cnt.data_ptr(), L, q, stream())
    np.testing.assert_array_equal(host(cnt, np.uint32), oracle.bicounts(mem, L, q, nseq=N))

    out = empty((np_, qq), np.float32)
    nb = int(_lib.query("mi3_weighted_marg_workspace", L, q, N))
    ws = empty((nb // 8 + 1,), np.int64)
    _lib.call("mi3_weighted_marg", dw.data_ptr(), dm.data_ptr(), B, N, out.data_ptr(), L, q, None, ws.data_ptr(), nb,
              stream())
    ref = oracle.weighted_marg_f64(w, np.ascontiguousarray(mem[:, :N]), L, q)
    # each weight rounded to 2^-17 of the largest at worst
    assert (np.abs(host(out) - ref) / ref.sum(axis=1, keepdims=True)).max() < 1e-5
    if 4 <= q <= 32 and N > 33:
        # the tensor-core form has the same scale, so the same integers
        out2 = empty((np_, qq), np.float32)
        st = empty((1,), np.int32)
        nb = int(_lib.query("mi3_weighted_marg_tc_workspace", L, q))
        ws = empty((nb // 8 + 1,), np.int64)
        _lib.call("mi3_weighted_marg_tc", dw.data_ptr(), dm.data_ptr(), B, N, out2.data_ptr(), L, q, ws.data_ptr(), nb,
                  st.data_ptr(), stream())
        assert int(host(st)[0]) == 0
        np.testing.assert_array_equal(host(out2), host(out))


@pytest.mark.parametrize("q", QS)
@pytest.mark.parametrize("L", [15, 31, 33, 65])
def test_equal_sequences_have_equal_energies(cuda, L, q):
    """A sequence's energy depends on its residues alone, not on the lane or the
    chunk that sums it: copies tie, and share their average rank."""
    rng = np.random.default_rng(100 * q + L)
    J, kinds, N = random_model(L, q, q + L), 5, 4101
    which = rng.integers(0, kinds, size=N)
    which[:160] = np.repeat(np.arange(kinds), 32)  # each in every lane
    mem = oracle.pack_seqs(rng.integers(0, q, size=(kinds, L)).astype("<u1")[which])
    dm, dJ = dev(mem), dev(J)
    E, r = empty((N,), np.float32), empty((N,), np.float32)
    ws = empty((N + 1,), np.int64)
    _lib.call("mi3_energies", dJ.data_ptr(), dm.data_ptr(), N, N, E.data_ptr(), L, q, ws.data_ptr(), ws.numel() * 8,
              stream())
    e = host(E)
    for k in range(kinds):
        assert np.unique(e[which == k]).size == 1
    ws = empty((int(_lib.query("mi3_rank_workspace", N)) // 8 + 2,), np.int64)
    _lib.call("mi3_rank_average", E.data_ptr(), N, r.data_ptr(), ws.data_ptr(), ws.numel() * 8, stream())
    np.testing.assert_array_equal(host(r), oracle.rank_average(e).astype("<f4"))


@pytest.mark.parametrize("q", [3, 5, 8, 21])
def test_residues_past_the_alphabet_count_as_the_last(cuda, q):
    """Invalid residues (>= q) are clamped, as the pair kernels always did."""
    L, N = 37, 600
    rng = np.random.default_rng(q)
    seqs = rng.integers(0, q, size=(N, L)).astype("<u1")
    bad = seqs.copy()
    at = rng.random((N, L)) < 0.02
    seqs[at] = q - 1
    bad[at] = rng.integers(q, 256, size=int(at.sum()))
    res = []
    for s in (seqs, bad):
        cnt = empty((L * (L - 1) // 2, q * q), np.uint32)
        dm = dev(oracle.pack_seqs(s))
        _lib.call("mi3_bicounts", dm.data_ptr(), N, N, cnt.data_ptr(), L, q, stream())
        res.append(host(cnt, np.uint32))
    np.testing.assert_array_equal(res[1], res[0])


@pytest.mark.parametrize("L,q", [(48, 4), (93, 4), (232, 21), (187, 8), (512, 21)])
def test_weighted_workspace_serves_fewer_sequences(L, q):
    last = 0
    for n in sorted({512 * k for k in range(1, 2100, 7)}):
        need = int(_lib.query("mi3_weighted_marg_workspace", L, q, n))
        assert need >= last
        last = need
