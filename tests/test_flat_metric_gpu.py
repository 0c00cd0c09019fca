"""The Minkowski kernels against the general metric's on the same metric: a
Kerr-Schild handle whose geometry is set to Minkowski runs every term the
Minkowski kernels drop (products with the metric's zeros and ones).

In the FP64 parity form the two give the same bits (adding a zero and
multiplying by one are exact; with conduction or viscosity too); in the mixed
form the compiler contracts the two differently, so they agree to rounding:
1e-12 of each variable's scale, some 1e3 operations at 1e-16 on these
well-conditioned states (largest seen: 3.4e-14, with extended MHD 3.2e-14).  A non-finite value, which a zero term spreads
(0 x Inf is NaN), is lost in the same zones.
"""
import numpy as np
import pytest

from grim_b200 import config as C
from grim_b200 import problems as PR
from tests.helpers import interior, scaled_err

pytestmark = pytest.mark.gpu


def _config(dim, emhd, scheme, solver, **kw):
    # sizes with a remainder in every lane split (31 faces of X1 per warp, 7
    # of X2 / X3), the smallest an active direction may have along X3
    n = {1: (45, 1, 1), 2: (37, 12, 1), 3: (34, 9, 4)}[dim]
    return PR.fast_mode_config(N=32, N1=n[0], N2=n[1], N3=n[2], dim=dim, conduction=emhd, viscosity=emhd,
                               reconstruction=scheme, riemannSolver=solver, dt=2e-3, **kw)


def _state(cfg, seed=11):
    rng = np.random.default_rng(seed)
    dof, nf = C.var_counts(cfg)
    P = np.zeros((dof,) + tuple(reversed(C.total_dims(cfg))))
    base = [1.0, 2.0, 0.1, -0.05, 0.02] + [0.01] * (nf - 5) + [0.1, 0.3, -0.2]
    for v in range(dof):
        P[v] = base[v] * (1. + 0.2 * rng.uniform(-1., 1., P.shape[1:]))
    return P


def _pair(cfg, mode, P, steps=2):
    """(Minkowski kernels', general kernels') primitives after the steps."""
    from grim_b200.timestepper import timeStepper
    out = []
    for metric in (C.MINKOWSKI, C.MODIFIED_KERR_SCHILD):
        ts = timeStepper(dict(cfg, metric=metric, newtonMode=mode, perZoneConvergence=int(mode != 0)))
        if metric == C.MODIFIED_KERR_SCHILD:
            eta = np.zeros((4, 4) + ts.zshape)
            for m in range(4):
                eta[m, m] = -1. if m == 0 else 1.
            one = np.ones(ts.zshape)
            for loc in (C.CENTER, C.LEFT, C.RIGHT, C.TOP, C.BOTTOM):
                ts.setGeometry(loc, eta, eta, one, one, gamma=np.zeros((64,) + ts.zshape))
        ts.primOld.setVars(P)
        ts.primOld.communicate()
        ts.timeSteps(steps)
        out.append(interior(cfg, ts.primOld.getVars()))
    return out


@pytest.mark.parametrize("scheme", [C.MINMOD, C.WENO5, C.PPM, C.MP5])
@pytest.mark.parametrize("solver", [C.HLL, C.LOCAL_LAX_FRIEDRICH])
@pytest.mark.parametrize("emhd", [0, 1])
@pytest.mark.parametrize("dim", [1, 2, 3])
def test_minkowski_kernels_match_the_general_ones(dim, emhd, solver, scheme):
    cfg = _config(dim, emhd, scheme, solver)
    P = _state(cfg)
    a, b = _pair(cfg, C.NEWTON_PARITY_FD64, P)
    assert np.all(np.isfinite(b)) and np.array_equal(a, b)
    tol = dict(nonlinearsolve_rtol=1e-12, nonlinearsolve_atol=1e-28, nonlinearsolve_ulps=8., maxNonLinearIter=6)
    a, b = _pair(_config(dim, emhd, scheme, solver, **tol), C.NEWTON_MIXED32, P)
    assert scaled_err(a, b) <= 1e-12


@pytest.mark.parametrize("mode", [C.NEWTON_PARITY_FD64, C.NEWTON_MIXED32])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("solver", [C.HLL, C.LOCAL_LAX_FRIEDRICH])
def test_a_non_finite_value_is_lost_in_the_same_zones(solver, value, mode):
    cfg = _config(2, 0, C.MINMOD, solver)
    for var in ("U1", "U2", "U3", "B1", "B2"):
        P = _state(cfg)
        P[C.var_index(cfg)[var], 0, 8, 19] = value
        a, b = _pair(cfg, mode, P, steps=1)
        lost = ~np.all(np.isfinite(b), axis=0)
        assert lost.any() and not lost.all()
        assert np.array_equal(~np.all(np.isfinite(a), axis=0), lost), var
