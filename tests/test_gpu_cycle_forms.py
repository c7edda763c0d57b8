"""GPU check of the FP32 V-cycle's kernels (the coarse tail's forms, levels above it in
short and long marches, even and uneven axes) against the FP64 ones: one V-cycle of the
mixed mode leaves the residual that one FP64 V-cycle of the plain mode leaves on the
same problem.

Both run the same Chebyshev cycle from the same start, so they differ by the FP32
rounding of the correction alone: about 1e-5 of the starting residual (cycle
depth times 2^-24, times the cancellation of the residual, at most 1e3), which is
at most 1e-3 of the residual a cycle leaves (contraction at least 1e-2).  A wrong
halo plane or image changes the residual by its own order."""
import math

import numpy as np
import pytest

from saras_gb300 import Solver, _abi as F
from tests import _cases as C

pytestmark = pytest.mark.gpu

# kind, grid indices, depth, pre / post sweeps, sweeps below the finest level (0: the same)
CASES = [("tgv", (6, 6, 6), 4, 3, 3, 0), ("tgv", (6, 6, 6), 5, 2, 2, 0), ("ldc", (6, 6, 6), 4, 3, 3, 0), ("ldc", (5, 5, 5), 3, 2, 1, 0),
         ("tgv", (5, 5, 5), 4, 3, 2, 0), ("rbc", (6, 6, 5), 4, 3, 3, 0), ("rbc", (7, 7, 6), 5, 3, 3, 2), ("ldc", (7, 5, 5), 3, 3, 3, 0),
         ("tgv", (7, 7, 7), 6, 4, 3, 0), ("ldc", (6, 5, 6), 4, 2, 2, 8), ("ldc", (5, 6, 6), 3, 3, 3, 0)]


def one_cycle(kind, ind, depth, pre, post, coarse, mode):
    p = C.CASES[kind](ind=ind if kind == "rbc" else ind[0], depth=depth)
    p.xInd, p.yInd, p.zInd = ind
    if kind == "ldc":
        p.Lx, p.Ly, p.Lz = (2.0 ** (i - 5) for i in ind)      # equal spacings
    p.mgMode = mode
    p.mgTarget, p.mgMaxCycles, p.mixedCycles = 1e-13, 1, 1
    p.preSmooth, p.postSmooth, p.coarseSmooth = pre, post, coarse
    p.smoother, p.jacobiWeight = F.SMOOTHER_CHEBYSHEV, 6.0 / 7.0
    p.fastKernels = 1
    g = Solver(p)
    C.initialise(g, p, kind)
    rng = np.random.default_rng(23)
    for f in (F.FIELD_VX, F.FIELD_VY, F.FIELD_VZ):
        g.set(f, g.get(f) + 0.1 * rng.standard_normal(g.dims(f)))
        g.apply_bc(f)
    status, st = g.time_advance()
    assert status == F.NOT_CONVERGED and st.vcycles == 1
    return st.fine_residual, st.guess_residual


@pytest.mark.parametrize("kind,ind,depth,pre,post,coarse", CASES)
def test_one_cycle_leaves_the_fp64_residual(kind, ind, depth, pre, post, coarse):
    r32, s32 = one_cycle(kind, ind, depth, pre, post, coarse, F.MG_MIXED)
    r64, s64 = one_cycle(kind, ind, depth, pre, post, coarse, F.MG_PLAIN_TARGET)
    assert math.isclose(s32, s64, rel_tol=1e-9)
    assert math.isclose(r32, r64, rel_tol=1e-3), (r32, r64)
