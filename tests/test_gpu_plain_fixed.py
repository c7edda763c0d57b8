"""GPU check of where the plain target mode leaves its fixed-point levels (plain_fixed):
solves of given right-hand sides and starts against the FP64 levels.  A context that
asks for an extrapolated guess runs the FP64 levels; its first solve has no history, so
it starts from the given Pp too."""
import numpy as np
import pytest

import saras_gb300 as S
from saras_gb300 import _abi as F
from tests import _cases as C

pytestmark = pytest.mark.gpu


def solver(fp64, ind=5, depth=3, pre=2, post=2, smoother=F.SMOOTHER_CHEBYSHEV, target=1e-8, cycles=100):
    p = C.tgv(ind=ind, depth=depth)
    p.Lx = p.Ly = p.Lz = 1.0
    p.mgMode, p.mgTarget, p.mgMaxCycles = F.MG_PLAIN_TARGET, target, cycles
    p.smoother, p.jacobiWeight, p.coarseCycles = smoother, 6.0 / 7.0, 1
    p.preSmooth, p.postSmooth = pre, post
    g = S.Solver(p)
    if fp64:
        g.set_guess_mode(F.GUESS_EXTRAPOLATE)
    return g


def lap(P):
    """Sum of the six neighbours less six times the point on the periodic N^3 box."""
    return sum(np.roll(P, s, d) for d in range(3) for s in (1, -1)) - 6 * P


def solve(g, P, b):
    """(status, V-cycles, Pp) of the solve of l lap(Pp) = b from P, l = N^2."""
    n = b.shape[0]
    i = np.arange(-1, n + 2) % n
    g.set(F.FIELD_PP, P[np.ix_(i, i, i)])
    g.set(F.FIELD_MGRHS, b[np.ix_(i, i, i)])
    status, cycles = 0, None
    try:
        cycles, _ = g.mg_solve()
    except S.SarasError as e:
        status = e.status
    return status, cycles, g.get(F.FIELD_PP)[1:n + 1, 1:n + 1, 1:n + 1]


@pytest.mark.parametrize("k,amplitude", [((2, 2, 2), 57.25), ((1, 2, 2), 57.0)])
def test_residual_too_large_for_a_plane_sum(k, amplitude):
    """A smooth start residual of 2^57 units: the 17^3 level's, eight times as large in its unit and
    hardly smaller after its sweep, passes 2^59, where the sum of 16 wraps.  The solve runs on the
    FP64 levels, bit for bit."""
    n = 32
    x = 2 * np.pi * np.arange(n) / n
    m = np.cos(k[0] * x)[:, None, None] * np.cos(k[1] * x)[None, :, None] * np.cos(k[2] * x)[None, None, :]
    P = 0.75 * np.cos(x)[:, None, None] * np.ones((n, n, n))       # a unit of 2^-58
    b = n * n * (lap(P) + 2.0 ** (amplitude - 58) * m)
    for cycles in (1, 2, 100):
        out = [solve(solver(fp64, pre=1, post=2, smoother=F.SMOOTHER_JACOBI, cycles=cycles), P, b) for fp64 in (0, 1)]
        assert out[0][:2] == out[1][:2] and (out[0][0] == 0) == (cycles == 100)
        assert np.array_equal(out[0][2], out[1][2]), cycles
