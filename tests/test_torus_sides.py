"""The torus's boundary pass on every accepted choice of X1 sides.

The reference fills the ghost zones and then checks the inflow in the X1
ghosts (boundary.cpp:5-241, torus/problem.cpp:941-1044).  One launch may do
both only where no ghost zone's fill reads a zone the check rewrites; the rule
that picks it (torus_fill_checks) is compared here with that condition over all
sides, and the pass itself with a restatement on sides of either kind.
"""
import itertools
import os
import subprocess

import numpy as np
import pytest

from grim_b200 import config as C
from grim_b200.build import COMMON, CSRC, NVCC
from grim_b200.problems import torus as T

SIDES = (C.PERIODIC, C.OUTFLOW, C.MIRROR, C.EXCHANGE)
NG = 3


def _source(x, n, lo, hi):
    """The index along one direction that the fill of index x reads."""
    if C.PERIODIC in (lo, hi) or NG <= x < n + NG:
        return x  # grid::communicate fills a periodic direction, at the end of the stage
    side = lo if x < NG else hi
    if side == C.EXCHANGE:
        return x
    if side == C.MIRROR:
        return 2 * NG - 1 - x if x < NG else 2 * (n + NG) - 1 - x
    return NG if x < NG else n + NG - 1


def _map(n, lo, hi):
    return [_source(x, n, lo, hi) for x in range(n + 2 * NG)]


def test_one_launch_only_where_no_fill_reads_a_checked_zone(tmp_path):
    src = tmp_path / "rule.cu"
    src.write_text('#include <cstdio>\n#include <cstring>\n#include "launch.h"\n'
                   "int main() {\n  for (int lo = 0; lo < 5; lo++)\n    for (int hi = 0; hi < 5; hi++) {\n"
                   "      grim::DevCfg c;\n      memset(&c, 0, sizeof c);\n      c.bc[0] = lo;\n      c.bc[1] = hi;\n"
                   '      printf("%d %d %d\\n", lo, hi, grim::torus_fill_checks(c) ? 1 : 0);\n    }\n}\n')
    subprocess.run([NVCC] + COMMON + ["-I", CSRC, str(src), "-o", str(tmp_path / "rule")], check=True)
    rows = subprocess.run([str(tmp_path / "rule")], check=True, capture_output=True, text=True).stdout.split("\n")
    rule = {tuple(map(int, r.split()[:2])): r.split()[2] == "1" for r in rows if r}
    n1, n3 = 5, 4
    together = 0
    for lo1, hi1 in itertools.product(SIDES, SIDES):
        reads = False  # over all X3 sides: does a fill read an X1 ghost of another zone
        m1 = _map(n1, lo1, hi1)
        for lo3, hi3 in itertools.product(SIDES, SIDES):
            for i, k in itertools.product(range(n1 + 2 * NG), range(n3 + 2 * NG)):
                si, sk = m1[i], _map(n3, lo3, hi3)[k]
                reads = reads or ((si, sk) != (i, k) and not NG <= si < n1 + NG)
        assert not (rule[lo1, hi1] and reads), (lo1, hi1)
        together += rule[lo1, hi1]
    assert together and rule[C.OUTFLOW, C.OUTFLOW]  # the torus's own sides take one launch


def _inflow(cfg, geo, P):
    """inflowCheck (torus/problem.cpp:941-1044) on the X1 ghost columns."""
    n1 = cfg["N1"]
    gcov = np.asarray(geo["gCov"])[1:, 1:]
    shift = np.asarray(geo["gCon"])[0, 1] * np.asarray(geo["alpha"])
    for cols in (range(NG), range(n1 + NG, n1 + 2 * NG)):
        for i in cols:
            u = P[2:5, :, :, i]
            g = gcov[..., i]
            u = u / np.sqrt(1. + np.einsum("akj,bkj,abkj->kj", u, u, g))
            u[0] = np.minimum(shift[..., i], u[0]) if i < NG else np.maximum(shift[..., n1 + NG - 1], u[0])
            v2 = np.einsum("akj,bkj,abkj->kj", u, u, g)
            v2 = np.clip(v2, 1e-13, 1. - 1. / cfg["MaxLorentzFactor"] ** 2)
            P[2:5, :, :, i] = u / np.sqrt(1. - v2)


@pytest.mark.gpu
@pytest.mark.parametrize("emhd", [False, True])
@pytest.mark.parametrize("x3", [C.OUTFLOW, C.MIRROR, C.PERIODIC])
@pytest.mark.parametrize("x1", [(C.OUTFLOW, C.OUTFLOW), (C.EXCHANGE, C.EXCHANGE), (C.PERIODIC, C.PERIODIC),
                                (C.MIRROR, C.EXCHANGE), (C.EXCHANGE, C.OUTFLOW)])
def test_boundary_pass_matches_a_restatement(x1, x3, emhd):
    from grim_b200.timestepper import timeStepper
    cfg = T.torus_config(N1=33, N2=17, N3=6, emhd=emhd, boundaryLeft=x1[0], boundaryRight=x1[1], boundaryBack=x3,
                         boundaryFront=x3, X1Start=np.log(4.), X1End=np.log(40.))  # X1 ghosts outside the horizon
    ts = timeStepper(cfg)
    geo = ts.getGeometry(C.CENTER)
    # every zone its own state, in- and outflowing, so that a wrong source or a
    # second check shows
    rng = np.random.default_rng(7)
    dof, nf = C.var_counts(cfg)
    P = np.zeros((dof,) + tuple(reversed(C.total_dims(cfg))))
    for v, base in enumerate([1., 0.1, 0.05, 0.02, 0.01] + [0.01] * (nf - 5) + [0.1, 0.03, -0.02]):
        P[v] = base * (rng.uniform(0.5, 1.5, P.shape[1:]) if v < 2 else rng.uniform(-1., 1., P.shape[1:]))
    for mode in (C.NEWTON_PARITY_FD64, C.NEWTON_MIXED32):
        ts.setNewtonMode(mode, int(mode != C.NEWTON_PARITY_FD64), 1e-10)
        ts.primOld.setVars(P)
        ts.stageSetup(C.HALF_STEP)
        got = ts.primOld.getVars()
        idx = [_map(cfg["N%d" % d], *s) for d, s in ((3, (x3, x3)), (2, (C.MIRROR, C.MIRROR)), (1, x1))]
        want = P[:, idx[0]][:, :, idx[1]][:, :, :, idx[2]].copy()
        _inflow(cfg, geo, want)
        # the rows the pole fix leaves alone
        rows = slice(NG + 2, cfg["N2"] + NG - 2)
        a, b = got[:, :, rows], want[:, :, rows]
        # velocities: a dozen operations on them and the metric, 1e-13 of the
        # zone's largest with the cancellation in g_ij u^i u^j; the rest are copies
        assert np.all(np.isfinite(b))
        scale = np.max(np.abs(b[2:5]), axis=0)
        assert np.max(np.abs(a[2:5] - b[2:5]) / scale) <= 1e-12
        other = [v for v in range(P.shape[0]) if not 2 <= v < 5]
        assert np.array_equal(a[other], b[other])
