"""Smoothing phases of no sweeps (V(0, n) and V(n, 0) cycles) against the oracle, bit
for bit: such a phase fills the ghosts and, where it starts a coarse level, leaves its
iterate 0."""
import numpy as np
import pytest

from oracle.oracle import Oracle
from saras_gb300 import Solver, _abi as F
from tests import _cases as C

pytestmark = pytest.mark.gpu


def cavity(ind, depth, gs, pre=3, post=3):
    p = C.ldc(ind=ind[0], depth=depth)
    p.xInd, p.yInd, p.zInd = ind
    p.gsSmooth, p.preSmooth, p.postSmooth = gs, pre, post
    p.vcCount = 4
    return p


def core(a, planar):
    return a[1:-1, 1:2, 1:-1] if planar else a[1:-1, 1:-1, 1:-1]


def two_steps(p):
    g, o = Solver(p), Oracle(p)
    rng = np.random.default_rng(3)
    for _ in range(2):                       # the second from the first one's level arrays
        for f in (F.FIELD_VX, F.FIELD_VZ):
            a = 0.1 * rng.standard_normal(g.dims(f))
            for s in (g, o):
                s.set(f, a)
                s.apply_bc(f)
        sg, stg = g.time_advance()
        so, sto = o.time_advance()
        assert sg == so == 0 and stg.vcycles == sto.vcycles
        assert np.array_equal(g.get(F.FIELD_PP), o.get(F.FIELD_PP))


@pytest.mark.parametrize("ind,depth", [((5, 5, 5), 2), ((6, 5, 4), 2), ((6, 0, 6), 3), ((8, 0, 8), 6)])
def test_gauss_seidel_phase_of_no_sweeps(ind, depth):
    p = cavity(ind, depth, 1)
    g, o = Solver(p), Oracle(p)
    rng = np.random.default_rng(1)
    for level in range(depth):               # levels in one CTA and beyond it
        a, r = rng.standard_normal(g.level_dims(level)), rng.standard_normal(g.level_dims(level))
        for s in (g, o):
            s.set_level(level, 1, r)
            s.set_level(level, 0, a)
            s.mg_smooth(level, 0)
            s.mg_restrict(level)             # reads the ghosts
        planar = not ind[1]
        assert np.array_equal(core(g.get_level(level, 0), planar), core(o.get_level(level, 0), planar)), level
        assert np.array_equal(core(g.get_level(level + 1, 1), planar), core(o.get_level(level + 1, 1), planar)), level


@pytest.mark.parametrize("ind,depth", [((5, 5, 5), 2), ((6, 0, 6), 4)])
@pytest.mark.parametrize("pre,post", [(0, 3), (3, 0), (0, 1)])
def test_gauss_seidel_cycle(ind, depth, pre, post):
    two_steps(cavity(ind, depth, 1, pre, post))


@pytest.mark.parametrize("pre,post", [(0, 3), (0, 1), (3, 0)])
def test_jacobi_cycle(pre, post):
    two_steps(cavity((5, 5, 5), 2, 0, pre, post))


@pytest.mark.parametrize("depth", [2, 4])    # levels of their own, and a tail from 9^3 down
def test_target_cycle(depth):
    """V(0, 3) cycles of the target modes: each one starts the coarse levels from 0, so the FP32
    and the FP64 cycles leave the same residual, up to FP32's rounding of a correction (1e-5 of the
    residual before it, and a cycle reduces that by 100 at most), and reduce it each time."""
    left = {}
    for mode in (F.MG_PLAIN_TARGET, F.MG_MIXED):
        for cycles in (1, 2, 3):
            p = cavity((5, 5, 5), depth, 0, 0, 3)
            p.mgMode, p.mgTarget, p.mgMaxCycles, p.mixedCycles = mode, 1e-13, cycles, 1
            p.smoother, p.jacobiWeight = F.SMOOTHER_JACOBI, 6.0 / 7.0
            g = Solver(p)
            rng = np.random.default_rng(3)
            for f in (F.FIELD_VX, F.FIELD_VZ):
                g.set(f, 0.1 * rng.standard_normal(g.dims(f)))
                g.apply_bc(f)
            status, st = g.time_advance()
            assert status == F.NOT_CONVERGED and st.vcycles == cycles
            left[mode, cycles] = st.fine_residual
    for cycles in (1, 2, 3):
        a, b = left[F.MG_PLAIN_TARGET, cycles], left[F.MG_MIXED, cycles]
        assert abs(a - b) <= 1e-3 * a, left
        assert cycles == 1 or a < 0.5 * left[F.MG_PLAIN_TARGET, cycles - 1], left
