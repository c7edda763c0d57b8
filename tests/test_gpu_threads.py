"""GPU check of two solvers in two host threads whose launches of one kernel ask for
different amounts of dynamic shared memory: the kernel's limit on the device is shared
by all of them."""
import threading

import numpy as np
import pytest

import saras_gb300 as S
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
