"""GPU check of saras_cn_solve_noalloc's batches of sweeps between waits against
saras_cn_solve, which waits after every sweep: solves of one sweep to several batches, on
both sides of the field size up to which it batches."""
import ctypes

import numpy as np
import pytest

import saras_gb300 as S
from saras_gb300 import _abi as F
from tests import _cases as C

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("ind", [(4, 4, 4), (5, 5, 6), (6, 6, 5)])
@pytest.mark.parametrize("fast", [0, 1])
@pytest.mark.parametrize("tol", [1.0, 1e-3, 1e-6, 1e-9, 1e-12])
def test_batched_sweeps_stop_where_single_ones_do(ind, fast, tol):
    p = C.ldc(ind=ind[0], depth=2, dt=0.05)
    p.xInd, p.yInd, p.zInd = ind
    p.fastKernels = fast
    p.cnTolerance = tol
    g = S.Solver(p)
    C.initialise(g, p, "ldc")
    rng = np.random.default_rng(3)
    v0 = g.get(F.FIELD_VX)
    rhs = v0 + 1e-2 * rng.standard_normal(v0.shape)
    g.set(F.FIELD_NSE_X, rhs)
    s, it, err = g.cn_solve(0)
    assert s == 0
    v = torch.tensor(v0, dtype=torch.float64, device="cuda:0").contiguous()
    r = torch.tensor(rhs, dtype=torch.float64, device="cuda:0").contiguous()
    torch.cuda.synchronize()
    n, e = ctypes.c_int(), ctypes.c_double()
    s = F.load().saras_cn_solve_noalloc(ctypes.byref(p), 0, ctypes.c_void_p(v.data_ptr()), ctypes.c_void_p(r.data_ptr()), None,
                                        ctypes.byref(n), ctypes.byref(e))
    assert s == 0 and n.value == it
    assert C.rel_err(v.cpu().numpy(), g.get(F.FIELD_VX)) <= 1e-10    # one arithmetic; the bound of the other checks of this call
    g.close()
