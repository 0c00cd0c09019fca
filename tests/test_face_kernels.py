"""The face-flux variants that launch one and the same kernel (face_kernel):
the autotuner times each kernel once, under the lowest of its numbers."""
import subprocess

import pytest

from grim_b200.build import COMMON, CSRC, NVCC

# variants per (unit, extended MHD, X1), and the kernels among them with a
# tensor map and without
KERNELS = {(1, 0, 1): (7, 4, 2), (1, 0, 0): (12, 8, 6), (0, 0, 1): (7, 7, 4), (0, 0, 0): (12, 12, 9),
           (1, 1, 1): (2, 2, 1), (1, 1, 0): (2, 2, 1), (0, 1, 1): (2, 2, 1), (0, 1, 0): (2, 2, 1)}


def test_every_variant_has_one_lowest_number(tmp_path):
    src = tmp_path / "t.cu"
    src.write_text('#include <cstdio>\n#include "launch.h"\nint main() {\n'
                   "  for (int fast = 0; fast < 2; fast++)\n    for (int emhd = 0; emhd < 2; emhd++)\n"
                   "      for (int dir = 0; dir < 3; dir++)\n        for (int tma = 0; tma < 2; tma++)\n"
                   "          for (int v = 0; v < (emhd ? 2 : dir ? 12 : 7); v++)\n"
                   '            printf("%d %d %d %d %d %d\\n", fast, emhd, dir, tma, v, '
                   "grim::face_kernel(fast, emhd, dir, v, tma));\n}\n")
    subprocess.run([NVCC] + COMMON + ["-I", CSRC, str(src), "-o", str(tmp_path / "t")], check=True)
    out = subprocess.run([str(tmp_path / "t")], check=True, capture_output=True, text=True).stdout
    table = {tuple(map(int, r.split()[:5])): int(r.split()[5]) for r in out.split("\n") if r}
    for (fast, emhd, dir_, tma, v), k in table.items():
        assert 0 <= k <= v and table[fast, emhd, dir_, tma, k] == k
    for fast, emhd, dir_, tma in {key[:4] for key in table}:
        mine = [k for key, k in table.items() if key[:4] == (fast, emhd, dir_, tma)]
        n, staged, plain = KERNELS[fast, emhd, int(dir_ == 0)]
        assert len(mine) == n and len(set(mine)) == (staged if tma else plain)


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [0, 3])
def test_autotune_picks_a_lowest_number_and_every_variant_gives_the_same_bits(mode):
    import numpy as np
    from grim_b200 import config as C
    from grim_b200 import problems as PR
    from grim_b200.timestepper import timeStepper
    mode = (C.NEWTON_PARITY_FD64, C.NEWTON_MIXED32)[mode == 3]
    cfg = PR.fast_mode_config(N=32, N1=34, N2=16, N3=8, dim=3, reconstruction=C.PPM, newtonMode=mode,
                              perZoneConvergence=int(mode != 0))
    rng = np.random.default_rng(1)
    P = np.zeros((8,) + tuple(reversed(C.total_dims(cfg))))
    for v, b in enumerate((1.0, 2.0, 0.1, -0.05, 0.02, 0.1, 0.3, -0.2)):
        P[v] = b * (1. + 0.1 * rng.uniform(-1., 1., P.shape[1:]))
    ts = timeStepper(cfg)
    ts.primOld.setVars(P)
    ts.primOld.communicate()
    fast = {0: {0, 1, 2, 3}, 1: {0, 1, 2, 3, 4, 5, 8, 9}}
    for d, (v, ms) in ts.autotune().items():
        assert ms > 0 and (mode == C.NEWTON_PARITY_FD64 or v in fast[int(d > 0)])
    ref = None
    for v in range(12):
        for d in range(3):
            ts.setFaceVariant(d, min(v, 6) if d == 0 else v)
        ts.primOld.setVars(P)
        ts.stageSetup(C.HALF_STEP)
        got = ts.stageGrid(1)
        if ref is None:
            ref = got
            # as many roundings apart as two compilations of a face may be: 1e-13
            # of the conserved variables' scale over a zone's width
            width = sum(cfg["N%d" % d] / (cfg["X%dEnd" % d] - cfg["X%dStart" % d]) for d in (1, 2, 3))
            tol = 1e-13 * 4 * np.max(np.abs(ts.stageGrid(0))) * width
        assert np.max(np.abs(got - ref)) <= (0. if mode == C.NEWTON_PARITY_FD64 else tol), v
