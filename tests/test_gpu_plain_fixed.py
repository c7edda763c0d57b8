"""GPU check of where the plain target mode leaves its fixed-point levels (plain_fixed):
solves of given right-hand sides and starts against the FP64 levels.  A context that
asks for an extrapolated guess runs the FP64 levels; its first solve has no history, so
it starts from the given Pp too."""
import math

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
    """(status, V-cycles, Pp, reported residual) of the solve of l lap(Pp) = b from P, l = N^2."""
    n = b.shape[0]
    i = np.arange(-1, n + 2) % n
    g.set(F.FIELD_PP, P[np.ix_(i, i, i)])
    g.set(F.FIELD_MGRHS, b[np.ix_(i, i, i)])
    status, cycles, res = 0, None, None
    try:
        cycles, res = g.mg_solve()
    except S.SarasError as e:
        status = e.status
    return status, cycles, g.get(F.FIELD_PP)[1:n + 1, 1:n + 1, 1:n + 1], res


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


def smooth(n, seed):
    """A few of the first waves, without a mean."""
    rng = np.random.default_rng(seed)
    x = 2 * np.pi * np.arange(n) / n
    b = np.zeros((n, n, n))
    for _ in range(6):
        k = rng.integers(0, 5, 3) + np.array([1, 0, 0])
        b += rng.standard_normal() * np.cos(k[0] * x[:, None, None] + k[1] * x[None, :, None] + k[2] * x[None, None, :] + 6 * rng.random())
    return b - b.mean()


@pytest.mark.parametrize("scale,target,fp64", [(0, 1e-8, False), (0, 1e-12, False), (10, 1e-12, False), (20, 1e-8, False), (20, 1e-12, True),
                                               (30, 1e-8, True), (40, 1e-8, True), (60, 1e-8, True)])
def test_start_far_above_the_solution(scale, target, fp64):
    """A start 2^scale times the solution's size: the solve meets its target (the exact residual of the
    returned Pp, in extended precision), on the FP64 levels where the start's unit is too coarse for it."""
    n = 32
    b, P = smooth(n, 2), 2.0 ** scale * 3.0 / n ** 2 * smooth(n, 3)
    out = [solve(solver(a, target=target), P, b) for a in (0, 1)]
    assert out[0][0] == out[1][0] == 0
    assert np.array_equal(out[0][2], out[1][2]) == fp64
    c = b.astype(np.longdouble) - b.astype(np.longdouble).mean()
    r = c - n * n * lap(out[0][2].astype(np.longdouble))
    assert np.max(np.abs(r)) <= target * np.max(np.abs(c)) * (1 + 1e-6)


@pytest.mark.parametrize("scale,target", [(0, 1e-12), (10, 1e-12), (20, 1e-8), (20, 1e-12), (30, 1e-8), (40, 1e-8)])
def test_start_far_above_the_solution_mixed(scale, target):
    """The same for the mixed mode's fixed-point refinement, which FP64 refinement takes over."""
    n = 32
    b, P = smooth(n, 2), 2.0 ** scale * 3.0 / n ** 2 * smooth(n, 3)
    g = solver(0)
    g.mg_set_mode(F.MG_MIXED, target, 100)
    status, _, p, _ = solve(g, P, b)
    c = b.astype(np.longdouble) - b.astype(np.longdouble).mean()
    r = c - n * n * lap(p.astype(np.longdouble))
    # FP64's own rounding of the residual it stops on: 14 terms of the solution's size
    slack = 14 * 2.0 ** -53 * n * n * np.max(np.abs(p))
    assert status == 0 and np.max(np.abs(r)) <= target * np.max(np.abs(c)) * (1 + 1e-6) + slack


@pytest.mark.parametrize("mode", [F.MG_PLAIN_TARGET, F.MG_MIXED])
def test_no_right_hand_side(mode):
    """0 on the right-hand side is exact in any unit: a constant Pp is its solution as it is."""
    g = solver(0)
    g.mg_set_mode(mode, 1e-8, 20)
    P = np.full((32, 32, 32), 0.7)
    status, cycles, p, res = solve(g, P, np.zeros(P.shape))
    assert (status, cycles, res) == (0, 0, 0.0) and np.array_equal(p, P)


def test_right_hand_side_below_the_unit():
    """Pp all one value, 2^70 times the right-hand side: in its unit the right-hand side is 0 and the
    residual too, which says nothing; FP64 levels cannot reduce it and say so."""
    b = smooth(32, 2)
    out = [solve(solver(a, cycles=20), np.full(b.shape, 2.0 ** 70), b) for a in (0, 1)]
    assert out[0][0] == out[1][0] == F.NOT_CONVERGED
    assert np.array_equal(out[0][2], out[1][2])


@pytest.mark.parametrize("depth", [1, 4])
def test_level_arrays_after_a_solve(depth):
    """The level calls read the FP64 values of what the fixed-point cycles left: level 0's right-hand
    side and solution exactly as given and returned, the residual they leave, and the levels below up
    to the FP64 residual's rounding (12 terms of the iterate's size).  A solve of the same problem
    after them has the same bits."""
    n = 32
    b, P = smooth(n, 2), 3.0 / n ** 2 * smooth(n, 3)
    g, h = solver(0, depth=depth), solver(1, depth=depth)
    (s, cycles, p, res), (t, _, q, _) = solve(g, P, b), solve(h, P, b)
    assert s == t == 0 and not np.array_equal(p, q)
    core = slice(1, n + 1)
    c = b - b.mean()
    unit = 2.0 ** -57 * np.max(np.abs(P)) * n * n                  # B's, at most
    assert np.max(np.abs(g.get_level(0, 1)[core, core, core] - c)) <= unit + 2.0 ** -52 * np.max(np.abs(c))
    assert np.array_equal(g.get_level(0, 0)[core, core, core], p)
    # (the reported residual is over both copies of a periodic plane, which a Gauss-Seidel coarse solve leaves unequal)
    assert abs(g.mg_compute_error(1) - res) <= 14 * 2.0 ** -53 * n * n * np.max(np.abs(p)) / np.max(np.abs(c))
    for level in range(1, depth + 1):
        for which in (0, 1):
            a, e = g.get_level(level, which), h.get_level(level, which)
            a, e = (v[1:-1, 1:-1, 1:-1] for v in (a, e))
            if which == 1:
                assert np.max(np.abs(a - e)) <= 14 * 2.0 ** -53 * n * n * np.max(np.abs(P) + np.abs(p)), level
            else:
                assert np.all(np.isfinite(a)) and np.max(np.abs(a)) <= 2 * np.max(np.abs(e)), level
    again = solve(g, P, b)
    assert again[:2] == (s, cycles) and np.array_equal(again[2], p)
    g.mg_set_mode(F.MG_REFERENCE)                                  # and another solver on the same arrays
    h.mg_set_mode(F.MG_REFERENCE)
    assert np.array_equal(solve(g, P, b)[2], solve(h, P, b)[2])


def test_network_that_does_not_fit():
    """A grid too shallow for the network: every call that needs it says so, and solves are as before."""
    b, P = smooth(32, 2), 3.0 / 32 ** 2 * smooth(32, 3)
    g, h = solver(0, depth=2), solver(0, depth=2)
    for call in (g.unet_shape, g.unet_shape, g.unet_collect, g.unet_collect, lambda: g.unet_train(1, 1e-3)):
        with pytest.raises(S.SarasError) as e:
            call()
        assert e.value.status == F.BAD_CONFIG
    p, q = solve(g, P, b), solve(h, P, b)
    assert p[:2] == q[:2] and np.array_equal(p[2], q[2])


def waves(p, seed):
    """A few of the first waves of the box on its padded points (whole waves on periodic axes, half waves between walls)."""
    rng = np.random.default_rng(seed)
    out = 0.0
    for _ in range(6):
        f = rng.standard_normal()
        for e, per, d in ((p.xInd, p.xPer, 0), (p.yInd, p.yPer, 1), (p.zInd, p.zPer, 2)):
            k = rng.integers(1, 4) * (2 if per else 1)
            f = f * np.cos(math.pi * k * np.arange(-1, 2 ** e + 2) / 2 ** e).reshape([-1 if q == d else 1 for q in range(3)])
        out = out + f
    return out


def problem(p):
    """A start and a right-hand side whose solution differs from it by a few hundredths (its residual, in
    units of 2^-57 of its maximum and less, stays where a level below can hold eight times as much)."""
    P, d = waves(p, 3), 0.03 * waves(p, 2)
    c = slice(1, -1)
    b = np.zeros(P.shape)
    b[c, c, c] = (2 ** p.xInd / p.Lx) ** 2 * sum(Q[2:, c, c] + Q[:-2, c, c] + Q[c, 2:, c] + Q[c, :-2, c] + Q[c, c, 2:] + Q[c, c, :-2] - 6 * Q[c, c, c]
                                               for Q in (P, d))
    return P, b


def one_cycle(make, fp64, pre, post, smoother):
    """(Pp before, Pp after) one V-cycle."""
    p = make()
    p.mgMode, p.mgTarget, p.mgMaxCycles = F.MG_PLAIN_TARGET, 1e-30, 1
    p.smoother, p.coarseCycles = smoother, 2
    p.preSmooth, p.postSmooth = pre, post
    g = S.Solver(p)
    if fp64:
        g.set_guess_mode(F.GUESS_EXTRAPOLATE)
    start, b = problem(p)
    g.set(F.FIELD_PP, start)
    g.set(F.FIELD_MGRHS, b)
    with pytest.raises(S.SarasError) as e:
        g.mg_solve()
    assert e.value.status == F.NOT_CONVERGED
    out = g.get(F.FIELD_PP)
    g.close()
    return start, out


@pytest.mark.parametrize("make,pre,post,smoother", [
    (lambda: C.tgv(ind=4, depth=1), 2, 1, 0),      # one 17^3 level above the coarsest, an odd sweep count
    (lambda: C.tgv(ind=5, depth=2), 2, 2, 1),      # two of them
    (lambda: C.ldc(ind=5, depth=3), 2, 2, 1),      # walls
    (lambda: C.rbc(ind=(5, 5, 4), depth=2), 1, 2, 1),
    (lambda: C.rbc(ind=(5, 5, 4), depth=2), 3, 0, 0),   # no sweep after the correction
    (lambda: C.tgv(ind=7, depth=5), 3, 3, 1),      # marches of eight planes
])
def test_cycle_runs_on_integers(make, pre, post, smoother):
    """The two arms run different levels (their last bits differ), and leave the same Pp up to the FP64
    arm's rounding: 12 terms of the iterate's size in the residual, which the coarse levels' inverse
    Laplacian amplifies by (N / pi)^2 at most, and a few more terms a sweep, not amplified; twice
    their sum, of the largest value on the way."""
    sa, a = one_cycle(make, False, pre, post, smoother)
    sb, b = one_cycle(make, True, pre, post, smoother)
    assert np.array_equal(sa, sb) and not np.array_equal(a, b)
    n = 2 ** make().xInd
    tol = 2.0 * (12.0 * (n / math.pi) ** 2 + 8.0 * (pre + post + 1)) * 2.0 ** -53
    assert np.max(np.abs(a - b)) <= tol * max(np.max(np.abs(sa)), np.max(np.abs(a)))


@pytest.mark.parametrize("bad", [math.nan, math.inf, -math.inf, None])
def test_values_out_of_range(bad):
    """Not a number or an infinity in the right-hand side, or (None) a solution a hundred times the
    start: the FP64 levels' result, bit for bit."""
    n = 32
    x = 2 * np.pi * np.arange(n) / n
    P = np.cos(x)[:, None, None] * np.ones((n, n, n))
    b = 100 * n * n * lap(P)
    assert np.max(np.abs(b)) / n ** 2 <= 4 * np.max(np.abs(P))     # a scale is taken
    if bad is not None:
        b[3, 4, 5] = bad
    out = [solve(solver(a, cycles=30), P, b) for a in (0, 1)]
    assert out[0][:2] == out[1][:2]
    assert np.array_equal(out[0][2], out[1][2], equal_nan=True)
