"""Small ideal-MHD grids run a stage's flux half and Newton in one launch and,
on periodic Minkowski grids, the stage's finish with them; profileSteps
launches the same pieces apart.  Both must give the same bits: the states and
their ghost zones, dt, time and the counters, eagerly and as a graph, on the
smallest grid an active direction may have (every zone then has a ghost image,
some two), on sizes that leave a block partly empty, and where only the launch
without the finish applies (an outflow side, Kerr-Schild with floors)."""
import numpy as np
import pytest

from grim_b200 import config as C
from grim_b200 import problems as PR
from grim_b200.problems import torus as T

pytestmark = pytest.mark.gpu

TOL = dict(nonlinearsolve_atol=1e-24, nonlinearsolve_rtol=1e-10, nonlinearsolve_ulps=8., maxNonLinearIter=4)


def _wave(cfg):
    rng = np.random.default_rng(2)
    P = np.zeros((8,) + tuple(reversed(C.total_dims(cfg))))
    for v, b in enumerate((1.0, 2.0, 0.1, -0.05, 0.02, 0.1, 0.3, -0.2)):
        P[v] = b * (1. + 0.1 * rng.uniform(-1., 1., P.shape[1:]))
    return P


def _flat(dim, n, **kw):
    return PR.fast_mode_config(N=32, N1=n[0], N2=n[1], N3=n[2], dim=dim, dt=1e-3, reconstruction=C.PPM, **TOL, **kw)


CASES = {
    "1d": lambda: _flat(1, (45, 1, 1)),
    "2d smallest": lambda: _flat(2, (4, 4, 1)),
    "2d ragged": lambda: _flat(2, (37, 12, 1)),
    "2d one side periodic": lambda: _flat(2, (16, 5, 1), boundaryTop=C.PERIODIC, boundaryBottom=C.OUTFLOW),
    "2d outflow": lambda: _flat(2, (33, 9, 1), boundaryTop=C.OUTFLOW, boundaryBottom=C.MIRROR),
    "3d": lambda: _flat(3, (10, 4, 5)),
    "dt from the half step": lambda: _flat(2, (20, 11, 1), elemOldFromFullStep=0),
    "torus": lambda: T.torus_config(N1=33, N2=17, N3=6, nonlinearsolve_atol=1e-24, nonlinearsolve_rtol=1e-10,
                                    nonlinearsolve_ulps=8.),
}


@pytest.mark.parametrize("mode", [C.NEWTON_MIXED32, C.NEWTON_TANGENT64])
@pytest.mark.parametrize("case", sorted(CASES))
def test_one_launch_gives_the_bits_of_the_pieces(case, mode):
    from grim_b200.timestepper import timeStepper
    cfg = dict(CASES[case](), newtonMode=mode, perZoneConvergence=1)
    ref = None
    for how in ("apart", "eager", "graph"):
        ts = timeStepper(cfg)
        if case == "torus":
            P, _ = T.torus_prims(cfg, ts.getGeometry(C.CENTER))
        else:
            P = _wave(cfg)
        ts.primOld.setVars(P)
        ts.primOld.communicate()
        ts.problemInit()
        ts.enableGraph(how == "graph")
        if how == "apart":
            ts.profileSteps(3)
        else:
            ts.timeSteps(3)
        st = ts.stats()
        got = [ts.primOld.getVars(), ts.primHalfStep.getVars(), ts.prim.getVars(), ts.stageGrid(0), ts.stageGrid(1),
               np.array([ts.time, ts.dt]), np.array(st["newtonIters"] + st["unconverged"] + [st["nonFinite"]]),
               np.array(ts.newtonHistogram())]
        assert np.all(np.isfinite(got[5])) and st["nonFinite"] == 0
        if ref is None:
            ref = got
        for k, (a, b) in enumerate(zip(got, ref)):
            assert np.array_equal(a, b, equal_nan=True), (how, k)
