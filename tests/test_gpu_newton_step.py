"""mi3_newton_step: the Newton phase through the one-call step equals the phase
through the separate calls, bit for bit."""
import numpy as np
import pytest

from mi3gpu_b200 import _lib, MCMCGPU, GPU_node, NewtonSteps, potts

pytestmark = pytest.mark.gpu


def _phase(L, q, N, reg, regarg, fused, onecall, mode="all"):
    rng = np.random.default_rng(L + q)
    g = MCMCGPU((0, 0), L, q, N, 512, None, 1024, 3)
    node = GPU_node([g])
    if not onecall:
        node.newtonStepper = lambda *a: None
        node.__class__ = type("Separate", (GPU_node,), {"newtonStepper": lambda self, *a: None})
    node.initJstep()
    node.setBuf("J", potts.synthetic_ground_truth(L, q, seed=L, contact_sigma=0.4))
    node.setSeqs("main", rng.integers(0, q, size=(N, L)).astype("<u1"))
    f = rng.uniform(0.5, 1.5, size=(L * (L - 1) // 2, q * q))
    node.setBuf("bi target", (f / f.sum(axis=1, keepdims=True)).astype("<f4"))
    p = NewtonSteps.Param()
    p.update(bimarg=None, gamma0=4e-3, newtonSteps=5, pcdamping=1e-3, fracNeff=0.1, nwalkers=N, reg=reg,
             regarg=regarg, beta=None, distribute_jstep=mode, L=L, q=q, device_resident=True)
    lines = []
    n, _, _ = NewtonSteps.iterNewton(p, None, node, lines.append, fused=fused)
    node.wait()
    seqbuf = "main" if mode == "all" else "large"
    out = [g.getBuf(b).read() for b in ("J", "dJ", "bi", "weightstats64", "minout", "E " + seqbuf,
                                        "weights" if mode == "all" else "weights large")]
    return n, out, [x for x in lines if "Neff" in x]


@pytest.mark.parametrize("L,q,N", [(20, 4, 1024), (33, 21, 1536)])
@pytest.mark.parametrize("reg,regarg", [(None, None), ("l1z", (2e-4,)), ("l2z", (1e-2,))])
def test_one_call_step_equals_separate_calls(cuda, L, q, N, reg, regarg):
    for fused in (True, False):
        a, b = _phase(L, q, N, reg, regarg, fused, True), _phase(L, q, N, reg, regarg, fused, False)
        assert a[0] == b[0] and a[2] == b[2]
        for x, y in zip(a[1], b[1]):
            np.testing.assert_array_equal(x, y)


def test_one_call_step_on_the_large_buffer(cuda):
    a, b = (_phase(20, 4, 1024, "l1z", (2e-4,), True, one, mode="head_gpu") for one in (True, False))
    for x, y in zip(a[1], b[1]):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("reg,regarg", [("SCADJ", (0.05, 0.5)), ("l1z", (2e-4,))])
def test_regularizer_arguments_may_be_an_array(cuda, reg, regarg):
    a, b = (_phase(20, 4, 1024, reg, r, True, True) for r in (regarg, np.array(regarg)))
    for x, y in zip(a[1], b[1]):
        np.testing.assert_array_equal(x, y)


def test_one_call_step_takes_only_what_it_does(cuda):
    g = MCMCGPU((0, 0), 12, 4, 512, 512, None, 1024, 3)
    g.initJstep()
    assert g.newtonStepper(1e-3, 1e-3, "X", (1.0,)) is None
    assert g.newtonStepper(1e-3, 1e-3, "l1z", (1.0, 2.0)) is None
    g.wmarg_kernel = "tc"
    assert g.newtonStepper(1e-3, 1e-3, None, ()) is None
    with pytest.raises(_lib.Mi3Error):
        _lib.call("mi3_newton_step", _lib.NewtonArgs(), 0.0, g._s)
