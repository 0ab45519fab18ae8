"""The fixed scratch of m16_maxflow_solve_static (25 MiB) holds the workspace of
every shape at its limits (262144 voxels, 4096 checks), thin volumes of many small
blocks included; the solve from it has the bits of one with a workspace."""
import ctypes

import numpy as np
import pytest

LIMIT, SCRATCH = 262144, 25 << 20


def test_every_shape_at_the_limits_fits():
    from miccai2016_gb300 import _native as N
    L = N.lib()
    p = N.CutParams(0.2, 0.11, 1e-4, 4094, 1, (ctypes.c_double * 3)(1, 1, 1))
    near = lambda lo, hi, offs: [2 ** k + o for k in range(lo, hi) for o in offs]
    rows, cols = list(range(1, 40)) + near(6, 19, (-1, 0, 1)), list(range(1, 300)) + near(9, 19, (-4, -3, -1, 0, 1, 4))
    worst = 0
    for d1 in rows:
        for d2 in cols:
            if d1 * d2 <= LIMIT:
                d0 = LIMIT // (d1 * d2)
                worst = max(worst, L.m16_maxflow_workspace_bytes(d0, d1, d2, ctypes.byref(p)))
    assert 88 * LIMIT < worst <= SCRATCH


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(1, 65536, 4), (2097, 5, 25), (64, 64, 64), (1, 1, 65536), (4681, 7, 8)])
@pytest.mark.parametrize("field", [False, True])
def test_thin_volumes_from_the_fixed_scratch(shape, field):
    import torch
    from miccai2016_gb300 import _native as N
    L = N.lib()
    g = torch.Generator(device="cuda")
    g.manual_seed(sum(shape))
    f = lambda *s: torch.rand(s, generator=g, device="cuda")
    img, quats, alpha, cs, ct, eigs = f(*shape), f(*shape, 3), f(*shape), f(*shape), f(*shape), 0.1 + f(*shape, 3)
    p = N.CutParams(0.2, 0.11, -1.0, 21, 5, (ctypes.c_double * 3)(1, 1, 1))
    L.m16_maxflow_solve_static.restype = ctypes.c_int
    L.m16_maxflow_solve_static.argtypes = L.m16_maxflow_solve.argtypes[:18] + [ctypes.c_void_p]
    sq = None if field else (ctypes.c_double * 3)(1.0, 0.3, 0.3)
    outs = []
    for static in (False, True):
        u = torch.empty(shape, device="cuda")
        it, n, res = ctypes.c_int32(0), ctypes.c_int32(0), (ctypes.c_double * 8)()
        args = [N.ptr(img), N.ptr(quats), sq, N.ptr(eigs) if field else None, N.ptr(alpha), 0.0, N.ptr(cs), N.ptr(ct), None,
                *shape, ctypes.byref(p), N.ptr(u), ctypes.byref(it), res, 8, ctypes.byref(n)]
        if static:
            st = L.m16_maxflow_solve_static(*args, N.stream_ptr())
        else:
            ws = N.workspace(L.m16_maxflow_workspace_bytes(*shape, ctypes.byref(p)))
            st = L.m16_maxflow_solve(*args, N.ptr(ws), ws.numel(), N.stream_ptr())
        assert st == N.M16_OK and it.value == 21 and n.value == 5
        outs.append((u.cpu().numpy().view(np.uint32), list(res[:5])))
    assert np.array_equal(outs[0][0], outs[1][0]) and outs[0][1] == outs[1][1]
