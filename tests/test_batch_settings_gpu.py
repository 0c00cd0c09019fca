"""What a batch step runs: the batch's own Newton on every problem, whatever
mode a problem's handle is given for steps of its own, and, as a graph, the
settings as they are now and not as they were when it was captured."""
import numpy as np
import pytest

from grim_b200 import config as C
from grim_b200 import problems as PR

pytestmark = pytest.mark.gpu

RTOL, ATOL = 1e-10, 1e-24


def _cfg(k):
    return PR.fast_mode_config(N=12 + k, reconstruction=(C.MINMOD, C.PPM, C.WENO5)[k % 3], nonlinearsolve_rtol=RTOL,
                               nonlinearsolve_atol=ATOL, maxNonLinearIter=5)


def _batch(n, graph):
    from grim_b200.timestepper import Batch
    cfgs = [_cfg(k) for k in range(n)]
    B = Batch(cfgs)
    B.setNewtonMode(C.NEWTON_MIXED32, RTOL)
    for k, (cfg, ts) in enumerate(zip(cfgs, B.problems)):
        P = PR.fast_mode_prims(cfg)
        X1, X2, _ = C.cell_centers(cfg)
        P[1] = P[1] + 1e-2 * np.sin(2 * np.pi * (X1 + 2 * X2))
        ts.primOld.setVars(P)
    B.enableGraph(graph)
    return B


def _states(B):
    B.synchronize()
    return [ts.primOld.getVars() for ts in B.problems] + [np.array([[ts.time, ts.dt] for ts in B.problems])]


def _same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("mode,perZone", [(C.NEWTON_TANGENT64, 1), (C.NEWTON_FD64_FAST, 0), (C.NEWTON_MIXED32, 3)])
def test_a_handles_own_newton_mode_leaves_the_batch_alone(mode, perZone, graph):
    A, B = _batch(4, graph), _batch(4, graph)
    A.timeSteps(2)
    B.timeSteps(1)
    B.problems[1].setNewtonMode(mode, perZone, 1e-2)
    B.timeSteps(1)
    assert _same(_states(A), _states(B))
    A.setNewtonMode(C.NEWTON_TANGENT64, RTOL)  # the batch's own mode is another matter
    B.setNewtonMode(C.NEWTON_TANGENT64, RTOL)
    A.timeSteps(1)
    B.timeSteps(1)
    assert _same(_states(A), _states(B))


@pytest.mark.parametrize("change", ["fixed dt", "parity stencil", "face variant"])
def test_a_setting_changed_after_the_capture_is_run(change):
    out = []
    for graph in (False, True):
        B = _batch(4, graph)
        B.timeSteps(2)
        for k, ts in enumerate(B.problems):
            if change == "fixed dt":
                ts.setFixedDt(True)
            elif change == "parity stencil" and k == 2:
                ts.setNewtonMode(C.NEWTON_PARITY_FD64, 0, RTOL)
            elif change == "face variant":
                ts.setFaceVariant(0, 1)
        B.timeSteps(2)
        out.append(_states(B))
    assert _same(*out)
    if change == "fixed dt":
        t = out[0][-1]
        B = _batch(4, False)
        B.timeSteps(4)
        assert not np.array_equal(_states(B)[-1], t)  # dt would have moved


@pytest.mark.parametrize("n", [1, 17, 20])
def test_more_problems_than_streams(n):
    """The eager step deals the problems to at most 16 streams; the captured
    one gives each a branch.  Each problem's states are those of the problem
    stepped alone, bit for bit."""
    from grim_b200.timestepper import timeStepper
    E, G = _batch(n, False), _batch(n, True)
    start = [ts.primOld.getVars() for ts in E.problems]
    E.timeSteps(3)
    G.timeSteps(3)
    e, g = _states(E), _states(G)
    assert _same(e, g)
    for k in range(n):
        ts = timeStepper(_cfg(k))  # as the batch made it: the first dt is the created handle's
        ts.setNewtonMode(C.NEWTON_MIXED32, 1, RTOL)
        ts.primOld.setVars(start[k])
        ts.timeSteps(3)
        assert np.array_equal(ts.primOld.getVars(), e[k]), k
