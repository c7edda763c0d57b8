"""GPU check of the plain target mode's fixed-point finest level (k_fx_sweep and its
companions) against the general FP64 level kernels: one V-cycle from the same state.  A
context that holds a network keeps b in level 0, so it takes the FP64 levels."""
import contextlib
import math

import numpy as np
import pytest

import saras_gb300 as S
from saras_gb300 import _abi as F
from tests import _cases as C

pytestmark = pytest.mark.gpu


def _one_cycle(make, general, pre, post, smoother):
    p = make()
    p.mgMode = F.MG_PLAIN_TARGET
    p.mgTarget = 1e-9
    p.mgMaxCycles = 100
    p.fastKernels = 2
    p.smoother = smoother
    p.coarseCycles = 2
    p.preSmooth, p.postSmooth = pre, post
    g = S.Solver(p)
    if general:
        with contextlib.suppress(Exception):   # (a grid too shallow for the network)
            g.unet_shape()
    C.initialise(g, p, {2: "tgv", 1: "ldc", 5: "rbc"}[p.probType])
    g.time_advance()                           # from Pp = 0: FP64 levels in both
    start = g.get(F.FIELD_PP)
    g.mg_set_mode(F.MG_PLAIN_TARGET, 1e-30, 1)
    s, st = g.time_advance()
    assert s == F.NOT_CONVERGED and st.vcycles == 1
    out = g.get(F.FIELD_PP)
    g.close()
    return start, out


@pytest.mark.parametrize("make,pre,post,smoother", [
    (lambda: C.tgv(ind=4, depth=1, dt=1e-3), 2, 1, 0),      # one 17^3 level above the coarsest, an odd sweep count
    (lambda: C.ldc(ind=5, depth=3, dt=1e-3), 2, 2, 1),      # walls
    (lambda: C.rbc(ind=(5, 5, 4), depth=2, dt=5e-4), 1, 2, 1),
    (lambda: C.rbc(ind=(5, 5, 4), depth=2, dt=5e-4), 3, 0, 0),   # no sweep after the correction
    (lambda: C.tgv(ind=7, depth=5, dt=5e-4), 3, 3, 1),      # marches of eight planes
])
def test_fixed_point_cycle_matches_fp64_cycle(make, pre, post, smoother):
    """The FP64 residual rounds 12 terms of the iterate's size, which the coarse levels'
    inverse Laplacian amplifies by (N / pi)^2 at most; a sweep rounds a few more terms, not
    amplified.  Twice their sum, of the largest value on the way."""
    sa, a = _one_cycle(make, False, pre, post, smoother)
    sb, b = _one_cycle(make, True, pre, post, smoother)
    assert np.array_equal(sa, sb)
    n = 2 ** make().xInd
    tol = 2.0 * (12.0 * (n / math.pi) ** 2 + 8.0 * (pre + post + 1)) * 2.0 ** -53
    assert np.max(np.abs(a - b)) <= tol * max(np.max(np.abs(sa)), np.max(np.abs(a)))
