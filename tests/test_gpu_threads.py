"""GPU check of solvers, in one host thread or in two, whose launches of one kernel ask
for different amounts of dynamic shared memory: the kernel's limit on the device is
shared by all of them."""
import threading

import numpy as np
import pytest

import saras_gb300 as S
from saras_gb300 import _abi as F
from tests import _cases as C

pytestmark = pytest.mark.gpu


def together(*work):
    errors = []

    def run(f):
        try:
            f()
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=run, args=(f,)) for f in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


def test_gauss_seidel_levels_of_two_solvers():
    def sweeps(ind, level):
        p = C.ldc(ind=ind, depth=2)
        p.gsSmooth = 1
        g = S.Solver(p)
        r = np.random.default_rng(1).standard_normal(g.level_dims(level))
        g.set_level(level, 1, r)
        for _ in range(4000):
            g.mg_smooth(level, 2)
        assert np.all(np.isfinite(g.get_level(level, 0)))
        g.close()

    together(lambda: sweeps(4, 1), lambda: sweeps(5, 1))          # 9^3 and 17^3


def test_coarsest_level_of_an_earlier_solver():
    """A coarsest level of 17^3 points (110 KB), then a solver with one of 5^3, then the first one's step."""
    p = C.tgv(ind=5, depth=1)
    p.mgMode, p.mgTarget, p.mgMaxCycles = F.MG_PLAIN_TARGET, 1e-8, 50
    first = S.Solver(p)
    C.initialise(first, p, "tgv")
    other = S.Solver(C.tgv(ind=4, depth=2))
    assert first.time_advance()[0] == 0
    other.close()
    first.close()


def test_convolutions_of_two_threads():
    def passes(cin, value):
        x = np.full((3, 3, 3, cin), value, dtype=np.float32)
        w = np.full((16, 27, cin), 0.125, dtype=np.float32)
        bits = S.to_bf16_bits(x)
        for _ in range(1500):
            y = S.conv3d_check(0, bits, None, w, None, 0, (3, 3, 3), cin, 16)
        assert np.all(y.reshape(3, 3, 3, 16)[1, 1, 1] == 0.125 * value * 27 * cin)   # exact: small integers over 8

    together(lambda: passes(16, 1.0), lambda: passes(96, 2.0))     # 24 and 140 KB
