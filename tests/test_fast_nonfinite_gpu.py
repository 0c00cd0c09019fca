"""Infinities and NaNs in the fast path's limiters.

The plain limiters take a NaN for positive and make 0 x Inf a NaN; a NaN made
on the GPU has its sign bit set, one made on the host has not.  A zone whose
stencil holds such a value must get the face values of the plain form, so the
face fluxes beside it are the parity path's: finite in the same places, and
there equal to the rounding of the two forms.
"""
import numpy as np
import pytest

from grim_b200 import config as C
from grim_b200 import problems as PR
from tests.helpers import interior

pytestmark = pytest.mark.gpu

NEGATIVE_NAN = np.uint64(0xFFF8000000000000).view(np.float64)


def _stepper(cfg, mode):
    from grim_b200.timestepper import timeStepper
    return timeStepper(dict(cfg, newtonMode=mode, perZoneConvergence=int(mode != 0)))


def _fluxes(ts, P):
    _, fl = ts.computeDivOfFluxes(P)
    return [interior(ts.cfg, f) for f in fl]


def _staged(ts, P, variant):
    """divF of a stage, the face kernels' variant per direction"""
    for d in range(3):
        ts.setFaceVariant(d, variant[d])
    ts.primOld.setVars(P)
    ts.stageSetup(C.HALF_STEP)
    return interior(ts.cfg, ts.stageGrid(1))


@pytest.mark.parametrize("value", [np.nan, NEGATIVE_NAN, np.inf, -np.inf])
@pytest.mark.parametrize("scheme", [C.MINMOD, C.PPM, C.WENO5, C.MP5])
@pytest.mark.parametrize("emhd", [0, 1])
def test_faces_beside_a_non_finite_value_are_the_plain_forms(emhd, scheme, value):
    cfg = PR.fast_mode_config(N=32, N1=37, N2=12, N3=4, dim=3, conduction=emhd, viscosity=emhd,
                              reconstruction=scheme)
    rng = np.random.default_rng(3)
    dof, nf = C.var_counts(cfg)
    shape = tuple(reversed(C.total_dims(cfg)))
    base = [1.0, 0.5, 0.1, -0.05, 0.02] + [0.01] * (nf - 5) + [0.1, 0.3, -0.2]
    clean = np.stack([b * (1. + 0.3 * rng.uniform(-1., 1., shape)) for b in base])
    plain, fast = _stepper(cfg, C.NEWTON_PARITY_FD64), _stepper(cfg, C.NEWTON_MIXED32)
    # as on finite data: a few hundred roundings of the largest flux or conserved
    # variable (WENO5: what its weights' rounding allows)
    tol = 3e-12 if scheme == C.WENO5 else 1e-13
    width = sum(cfg["N%d" % d] / (cfg["X%dEnd" % d] - cfg["X%dStart" % d]) for d in (1, 2, 3))
    u = np.max(np.abs(interior(cfg, plain.conserved(clean))))
    for var in range(dof):
        if var < 2 and np.isinf(value):
            continue  # the sound speed of an infinite rho or u is a NaN in the fast path: its own
        P = clean.copy()
        P[var, 4, 8, 20] = value
        P[var, 5, 9, 8] = value
        scale = u
        for d, (a, b) in enumerate(zip(_fluxes(fast, P), _fluxes(plain, P))):
            ok = np.isfinite(b)
            assert np.array_equal(np.isfinite(a), ok), (var, d)
            scale = max(scale, np.max(np.abs(b[ok])))
            assert np.max(np.abs(a[ok] - b[ok])) <= tol * scale, (var, d)
        b = _staged(fast, P, (0, 0, 0))
        a = _staged(fast, P, (1, 1, 1) if emhd else (2, 8, 8))  # staged through shared memory
        ok = np.isfinite(b)
        assert np.array_equal(np.isfinite(a), ok) and np.max(np.abs(a[ok] - b[ok])) <= 4 * tol * scale * width, var
        if emhd:
            # the gradients of u_mu and T: the explicit sources of q and deltaP, a
            # few hundred roundings apart
            a = interior(cfg, fast.stageGrid(2))[5:]
            _staged(plain, P, (0, 0, 0))
            b = interior(cfg, plain.stageGrid(2))[5:]
            ok = np.isfinite(b)
            assert np.array_equal(np.isfinite(a), ok), var
            assert np.max(np.abs(a[ok] - b[ok])) <= 1e-12 * np.max(np.abs(b[ok])), var
