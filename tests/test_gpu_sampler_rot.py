"""The rotated sampler (mi3_metropolis_rot) against the oracle and the row
kernel, bit for bit: every column mode and register class, tails of the last
chunk, partly filled CTAs, and couplings that leave many verdicts to the exact
sum."""
import numpy as np
import pytest

from oracle import oracle
from mi3gpu_b200 import _lib
from tests._util import dev, host, empty, stream, random_model

pytestmark = pytest.mark.gpu


def _table(J, L, q):
    T = empty((int(_lib.query("mi3_jrot_floats", L, q)),), np.float32)
    dJ = dev(J)
    _lib.call("mi3_unpack_j_rot", dJ.data_ptr(), T.data_ptr(), L, q, stream())
    host(T)  # waits: dJ may go
    return T


def _run(T, mem, st, pos, nsteps, L, q, wpc, betas=None, beta=1.0, lanes=0):
    N = mem.shape[1]
    m, s, status, dp = dev(mem), dev(st), empty((1,), np.int32), dev(pos)
    db = dev(betas) if betas is not None else None
    _lib.call("mi3_metropolis_rot", T.data_ptr(), s.data_ptr(), 0, dp.data_ptr(), nsteps,
              db.data_ptr() if db is not None else None, beta, m.data_ptr(), N, L, q, wpc, lanes,
              status.data_ptr(), stream())
    out = host(m, np.uint32), host(s, np.uint32)
    return (*out, int(host(status)[0]))


def _start(L, q, N, nsteps, seed):
    rng = np.random.default_rng(seed)
    mem = oracle.pack_seqs(rng.integers(0, q, size=(N, L)).astype("<u1"))
    st = oracle.init_rng(N, seed, 2 ** 63 // (2 * N))
    pos = np.concatenate([np.arange(L), rng.integers(0, L, size=nsteps)]).astype("<u4")[:nsteps]
    return mem, st, pos


# L at the ends of tails (8, 16, 32 columns) and chunks, per mode
SHAPES = [(2, 2, 32), (15, 2, 96), (16, 3, 64), (17, 3, 64), (48, 4, 160), (63, 4, 64), (65, 4, 64), (93, 4, 96),
          (129, 4, 64), (7, 5, 64), (34, 6, 64), (64, 7, 96), (66, 8, 64), (150, 8, 64), (9, 9, 32), (33, 12, 64),
          (40, 16, 64), (41, 20, 64), (48, 21, 64), (49, 21, 96)]


@pytest.mark.parametrize("sigma", [0.3, 3.0])
@pytest.mark.parametrize("L,q,N", SHAPES)
def test_rot_equals_oracle(cuda, L, q, N, sigma):
    """sigma = 3: bounds so wide that most verdicts take the exact sum."""
    J = random_model(L, q, L * q, sigma=sigma)
    nsteps = L + 37
    mem, st, pos = _start(L, q, N, nsteps, 5 * L + q)
    T = _table(J, L, q)
    o_mem, o_st = mem.copy(), st.copy()
    oracle.metropolis(J, o_st, pos, 0, nsteps, o_mem, L, q)
    for wpc, lanes in ((0, 0), (64, 1), (32, 2), (16, 4)):
        g_mem, g_st, status = _run(T, mem, st, pos, nsteps, L, q, wpc, lanes=lanes)
        assert status == 0
        np.testing.assert_array_equal(g_mem, o_mem)
        np.testing.assert_array_equal(g_st, o_st)


# register classes of the long shapes, 1, 2 and 4 lanes per walker, against the row
# kernel; 512 walkers so that both take them
@pytest.mark.parametrize("L,q", [(150, 4), (260, 4), (380, 3), (576, 2), (187, 8), (250, 6), (319, 5), (512, 8),
                                 (180, 21), (232, 21), (280, 21), (380, 10), (470, 21), (512, 21), (576, 16)])
def test_rot_equals_row_kernel(cuda, L, q):
    from mi3gpu_b200.potts import synthetic_ground_truth
    J = synthetic_ground_truth(L, q, seed=L + q)
    N, nsteps = 512, 200
    mem, st, pos = _start(L, q, N, nsteps, L)
    pos = np.random.default_rng(L).integers(0, L, size=nsteps).astype("<u4")
    betas = np.random.default_rng(q).uniform(0.5, 1.5, size=N).astype("<f4")
    stride = int(_lib.query("mi3_jrows_stride", L, q))
    Ju = empty((L, stride), np.float32)
    dJ = dev(J)
    _lib.call("mi3_unpack_j", dJ.data_ptr(), Ju.data_ptr(), L, q, stream())
    a_mem, a_st, status = dev(mem), dev(st), empty((1,), np.int32)
    dp, db = dev(pos), dev(betas)
    _lib.call("mi3_metropolis", Ju.data_ptr(), a_st.data_ptr(), 0, dp.data_ptr(), nsteps, db.data_ptr(), 1.0,
              a_mem.data_ptr(), N, L, q, status.data_ptr(), stream())
    T = _table(J, L, q)
    for lanes in (1, 2, 4):
        if lanes == 1 and L > 288 and q >= 8:
            continue  # no register class: rejected below
        g_mem, g_st, st_word = _run(T, mem, st, pos, nsteps, L, q, 0, betas=betas, lanes=lanes)
        assert st_word == 0 and int(host(status)[0]) == 0
        np.testing.assert_array_equal(g_mem, host(a_mem, np.uint32))
        np.testing.assert_array_equal(g_st, host(a_st, np.uint32))


@pytest.mark.parametrize("L,q", [(20, 4), (20, 8), (40, 21)])
def test_rot_infinite_and_huge_couplings(cuda, L, q):
    """Forbidden pairs (+inf, 1e30) and favoured ones: the bound is infinite,
    the exact sums decide, NaN differences included."""
    J = random_model(L, q, 3)
    rng = np.random.default_rng(q)
    for v in (np.inf, 1e30, -1e30):
        J[rng.integers(0, J.shape[0], 8), rng.integers(0, q * q, 8)] = v
    N, nsteps = 256, 120
    mem, st, pos = _start(L, q, N, nsteps, 2)
    o_mem, o_st = mem.copy(), st.copy()
    oracle.metropolis(J, o_st, pos, 0, nsteps, o_mem, L, q)
    g_mem, g_st, status = _run(_table(J, L, q), mem, st, pos, nsteps, L, q, 0)
    assert status == 0
    np.testing.assert_array_equal(g_mem, o_mem)
    np.testing.assert_array_equal(g_st, o_st)


@pytest.mark.parametrize("last", [False, True])
@pytest.mark.parametrize("L,q", [(20, 4), (20, 8), (40, 21)])
def test_rot_nan_couplings(cuda, L, q, last):
    """A NaN coupling, whatever its residues, leaves the verdicts of its letters
    to the exact sum, which rejects the moves that meet it."""
    J = random_model(L, q, 11)
    rng = np.random.default_rng(q)
    cells = rng.integers(0, q - 1, size=(2, 24)) if not last else np.full((2, 24), q - 1)
    J[rng.integers(0, J.shape[0], 24), cells[0] * q + cells[1]] = np.nan
    N, nsteps = 512, 6 * L
    mem, st, pos = _start(L, q, N, nsteps, 4)
    o_mem, o_st = mem.copy(), st.copy()
    oracle.metropolis(J, o_st, pos, 0, nsteps, o_mem, L, q)
    for lanes in (1, 2, 4):
        g_mem, g_st, status = _run(_table(J, L, q), mem, st, pos, nsteps, L, q, 0, lanes=lanes)
        assert status == 0
        np.testing.assert_array_equal(g_mem, o_mem)
        np.testing.assert_array_equal(g_st, o_st)


@pytest.mark.parametrize("L,q", [(20, 4), (21, 7), (40, 21)])
def test_rot_infinite_beta(cuda, L, q):
    """beta * dE overflows: the verdict hangs on the sign of dE.  Couplings in
    tenths, so that many differences are 0 but for the rounding of the sum."""
    rng = np.random.default_rng(q)
    J = (rng.integers(0, 4, size=(L * (L - 1) // 2, q * q)) / 10).astype("<f4")
    N, nsteps = 512, 4 * L
    mem, st, pos = _start(L, q, N, nsteps, 6)
    betas = np.resize(np.array([np.inf, 3e38, 1e38, -np.inf, 1.0], "<f4"), N)
    o_mem, o_st = mem.copy(), st.copy()
    oracle.metropolis(J, o_st, pos, 0, nsteps, o_mem, L, q, betas=betas)
    g_mem, g_st, status = _run(_table(J, L, q), mem, st, pos, nsteps, L, q, 0, betas=betas)
    assert status == 0
    np.testing.assert_array_equal(g_mem, o_mem)
    np.testing.assert_array_equal(g_st, o_st)


def test_rot_bad_site_reported_and_shapes_refused(cuda):
    L, q, N = 16, 4, 512
    T = _table(random_model(L, q, 6), L, q)
    mem, st, _ = _start(L, q, N, 3, 7)
    assert _run(T, mem, st, np.array([3, 99, 5], dtype="<u4"), 3, L, q, 0)[2] == 3  # MI3_STATUS_BAD_INPUT
    status, buf = empty((1,), np.int32), empty((16,), np.float32)
    for L, q, N, wpc, lanes in [(20, 22, 512, 0, 0), (577, 4, 512, 0, 0), (20, 4, 500, 0, 0), (20, 4, 1024, 40, 1),
                                (512, 21, 1024, 1024, 0), (20, 4, 512, 0, 3), (512, 21, 512, 0, 1)]:
        with pytest.raises(_lib.Mi3Error):
            _lib.call("mi3_metropolis_rot", buf.data_ptr(), buf.data_ptr(), 0, buf.data_ptr(), 1, None, 1.0,
                      buf.data_ptr(), N, L, q, wpc, lanes, status.data_ptr(), stream())


@pytest.mark.parametrize("L,q,kind", [(47, 4, "plan"), (48, 4, "rot"), (64, 6, "plan"), (400, 4, "plan")])
def test_untuned_choice_keeps_the_trajectories(cuda, L, q, kind):
    """Both sides of rot_default: the same walkers and generators as with the
    other kernel, bit for bit."""
    from mi3gpu_b200 import GPU_node, MCMCGPU
    N, out = 512, []
    for rot in (None, kind == "plan"):
        g = MCMCGPU((0, 0), L, q, N, 512, None, 1024, 3)
        assert g.sampler_kernel() == kind
        node = GPU_node([g])
        node.initMCMC(100)
        node.setSeqs("main", np.random.default_rng(5).integers(0, q, size=(N, L)).astype("<u1"))
        node.setBuf("J", random_model(L, q, 4))
        g.sampler_rot = rot
        node.runMCMC()
        out.append((node.collect("seq main"), g.getBuf("rngstates").read()))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])
