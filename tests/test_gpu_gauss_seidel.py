"""The pipelined Gauss-Seidel kernel (several lexicographic sweeps in flight)
against the oracle's sequential sweeps, bit for bit: smoothing phases of one to
seven sweeps on levels from three points an axis upwards, mirror and periodic
axes mixed, unequal axes, power-of-two and other metrics, 2D; and the coarsest
solve ending at its cap, part way (a tolerance met after some sweeps) and at
once."""
import numpy as np
import pytest

from oracle.oracle import Oracle
from saras_gb300 import Solver, _abi as F
from tests import _cases as C

pytestmark = pytest.mark.gpu

NNN, PPP, PPN, NPN, PNP = (0, 0, 0), (1, 1, 1), (1, 1, 0), (0, 1, 0), (1, 0, 1)
# grid indices, depth, periodic axes, length of the box
GRIDS = [((3, 3, 3), 2, NNN, 1.0), ((3, 3, 3), 2, PPP, 2.0), ((4, 4, 4), 2, NNN, 1.0), ((4, 4, 4), 2, PPP, 6.28), ((5, 4, 3), 2, PPN, 1.0),
         ((3, 4, 5), 2, PNP, 3.0), ((4, 5, 3), 2, NPN, 0.7), ((5, 5, 4), 2, PPN, 2.0), ((5, 5, 5), 2, PPP, 1.0), ((5, 5, 5), 2, NNN, 1.0),
         ((6, 5, 5), 3, NPN, 1.0), ((5, 6, 6), 3, PPP, 2.0),
         ((4, 0, 4), 2, NNN, 1.0), ((6, 0, 5), 3, NNN, 1.0), ((5, 0, 6), 2, (1, 0, 0), 1.5), ((7, 0, 7), 4, NNN, 1.0)]


def case(ind, depth, per, length, gs=1):
    p = C.base()
    p.probType, p.icType = (1, 0) if per == NNN else (2, 1)
    p.xPer, p.yPer, p.zPer = per
    p.xInd, p.yInd, p.zInd = ind
    p.Lx = p.Ly = p.Lz = length
    p.vcDepth = depth
    p.Re, p.tStp = 1000.0, 1e-3
    p.gsSmooth = gs
    return p


def core(a, planar):
    return a[1:-1, 1:2, 1:-1] if planar else a[1:-1, 1:-1, 1:-1]


@pytest.mark.parametrize("ind,depth,per,length", GRIDS)
def test_smoothing_sweeps(ind, depth, per, length):
    p = case(ind, depth, per, length)
    g, o = Solver(p), Oracle(p)
    rng = np.random.default_rng(7)
    for level in range(depth + 1):
        for count in (1, 2, 4, 7):
            a, r = rng.standard_normal(g.level_dims(level)), rng.standard_normal(g.level_dims(level))
            for s in (g, o):
                s.set_level(level, 1, r)
                s.set_level(level, 0, a)
                s.mg_smooth(level, count)
            x, y = g.get_level(level, 0), o.get_level(level, 0)
            assert np.array_equal(core(x, not ind[1]), core(y, not ind[1])), (level, count)
            g.mg_restrict(level) if level < depth else None    # reads the ghosts the sweeps left
            if level < depth:
                o.mg_restrict(level)
                assert np.array_equal(core(g.get_level(level + 1, 1), not ind[1]), core(o.get_level(level + 1, 1), not ind[1])), (level, count)


@pytest.mark.parametrize("make", ["ldc_d", "tgv_d", "rbc_d", "dirichlet", "2d257"])
def test_block_wavefront(make):
    """Levels beyond one CTA: stretched meshes, the Dirichlet check's walls and negated images, a large 2D level."""
    if make == "2d257":
        p = case((8, 0, 8), 6, NNN, 1.0)
    elif make == "dirichlet":
        p = case((5, 5, 5), 1, NNN, 1.0)
        p.testPoisson = 1
    else:
        p = C.CASES[make](ind=(6, 5, 5) if make == "rbc_d" else 5, depth=1 if make != "rbc_d" else 2)
        p.gsSmooth = 1
        p.vcDepth = 2
    g, o = Solver(p), Oracle(p)
    rng = np.random.default_rng(19)
    for level in (0, 1):
        for count in (1, 3, 4):
            a, r = rng.standard_normal(g.level_dims(level)), rng.standard_normal(g.level_dims(level))
            if make == "dirichlet":          # the walls' values come with a solve
                a[0], a[-1], a[:, 0], a[:, -1], a[:, :, 0], a[:, :, -1] = 0, 0, 0, 0, 0, 0
            for s in (g, o):
                s.set_level(level, 1, r)
                s.set_level(level, 0, a)
                s.mg_smooth(level, count)
            assert np.array_equal(core(g.get_level(level, 0), p.yInd == 0), core(o.get_level(level, 0), p.yInd == 0)), (level, count)


@pytest.mark.parametrize("tol", [1e-12, 1e-2, 0.3, 10.0])
@pytest.mark.parametrize("ind,depth,per,length", GRIDS)
def test_coarsest_solve(ind, depth, per, length, tol):
    """tol relative to the right-hand side's maximum: the cap, after some sweeps, after few, after one."""
    p = case(ind, depth, per, length, gs=0)
    dims = Solver(p).level_dims(depth)
    rng = np.random.default_rng(11)
    for kind in ("any", "compatible"):
        r = rng.standard_normal(dims)
        if kind == "compatible":                 # no part outside the operator's range: the sweeps converge
            w = [np.r_[0.0, 0.5, np.ones(n - 4), 0.5, 0.0] if n > 3 else np.array([0.0, 1.0, 0.0]) for n in dims]
            wt = w[0][:, None, None] * w[1][None, :, None] * w[2][None, None, :]
            r = r - np.sum(wt * r) / np.sum(wt)
        p.mgTolerance = tol * np.max(np.abs(r))
        g, o = Solver(p), Oracle(p)
        for s in (g, o):
            s.set_level(depth, 1, r)
            s.set_level(depth, 0, np.zeros(dims))
            s.mg_smooth(depth, -1)
        x, y = core(g.get_level(depth, 0), not ind[1]), core(o.get_level(depth, 0), not ind[1])
        assert np.array_equal(x, y), (kind, float(np.max(np.abs(x - y))))


@pytest.mark.parametrize("ind,depth,per,length", [((4, 4, 4), 2, NNN, 1.0), ((5, 5, 4), 2, PPN, 2.0), ((5, 0, 5), 3, NNN, 1.0)])
def test_solve_counts(ind, depth, per, length):
    """A whole solve: V-cycles and Gauss-Seidel sweeps of the coarsest level equal the oracle's."""
    p = case(ind, depth, per, length)
    p.vcCount = 6
    g, o = Solver(p), Oracle(p)
    rng = np.random.default_rng(13)
    for f in (F.FIELD_VX, F.FIELD_VZ):
        a = 0.1 * rng.standard_normal(g.dims(f))
        for s in (g, o):
            s.set(f, a)
            s.apply_bc(f)
    before = o.coarse_iters()
    sg, stg = g.time_advance()
    so, sto = o.time_advance()
    assert sg == so == 0 and stg.vcycles == sto.vcycles
    assert stg.coarse_iters == o.coarse_iters() - before
    assert np.array_equal(g.get(F.FIELD_PP), o.get(F.FIELD_PP))
