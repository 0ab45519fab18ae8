"""Check intervals longer than any solve, up to the largest that the 32-bit
`update` holds ("check iteration 0, then never again"): the solve runs its
num_iter iterations with the one residual of iteration 0, whether or not a bound
could stop it, with the launches timed or not, on both iteration paths."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("path", [0, 1])
@pytest.mark.parametrize("num_iter", [1, 6, 7])
@pytest.mark.parametrize("update", [2 ** 31 - 1, 2 ** 31 - 2, 2 ** 30, 1001])
@pytest.mark.parametrize("bound", [1e-30, -1.0])
def test_a_check_interval_beyond_the_solve(path, num_iter, update, bound):
    import torch
    from miccai2016_gb300 import _native as N
    L = N.lib()
    shape = (9, 18, 34)
    g = torch.Generator(device="cuda")
    g.manual_seed(num_iter)
    f = lambda *s: torch.rand(s, generator=g, device="cuda")
    img, quats, alpha, cs, ct = f(*shape), f(*shape, 3), f(*shape), f(*shape), f(*shape)
    outs = []
    for timed, upd in ((0, update), (1, update), (0, 7)):   # 7: checks iteration 0 alone in up to 7 iterations
        p = N.CutParams(0.2, 0.11, bound, num_iter, upd, (ctypes.c_double * 3)(1, 1, 1))
        ws = N.workspace(L.m16_maxflow_workspace_bytes(*shape, ctypes.byref(p)))
        u = torch.empty(shape, device="cuda")
        it, nres, res = ctypes.c_int32(0), ctypes.c_int32(0), (ctypes.c_double * 4)()
        st = N.SolveStats(timed, 0, 0, 0, 0.0, 0.0, path, 0)
        N.check("m16_maxflow_solve_ex", L.m16_maxflow_solve_ex(
            N.ptr(img), N.ptr(quats), (ctypes.c_double * 3)(1.0, 0.3, 0.3), None, N.ptr(alpha), 0.0, N.ptr(cs),
            N.ptr(ct), None, *shape, ctypes.byref(p), N.ptr(u), ctypes.byref(it), res, 4, ctypes.byref(nres),
            N.ptr(ws), ws.numel(), N.stream_ptr(), ctypes.byref(st)))
        assert it.value == num_iter and nres.value == 1
        outs.append((u.cpu().numpy().view(np.uint32), res[0]))
    for u, r in outs[1:]:
        assert np.array_equal(u, outs[0][0]) and r == outs[0][1]
