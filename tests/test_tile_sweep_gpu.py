"""The tile sweeps of the max-flow (csrc/tile_sweep.cuh): two iterations per
launch over tiles of 28 x 13 written columns in blocks of 32 x 16.

Sizes are the tiles' edges: one tile (32 columns, 16 rows), one column or row
more, the last column of the second and third tile, single planes.  Against
the oracle the tolerance is the max-flow's (1e-3 after a fixed iteration
count).  A stop after the first iteration of a pair has to give the bits of a
solve of that many iterations."""
import ctypes
import os
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(HERE, "golden"))

import inputs as I  # noqa: E402
from oracle import oracle as O  # noqa: E402

pytestmark = pytest.mark.gpu

U_TOL = 1e-3
E = 10 ** -1.5


def _inputs(seed, shape, supervised=False):
    rng = np.random.RandomState(seed)
    f = lambda lo, hi: rng.uniform(lo, hi, shape).astype(np.float32)
    return dict(img=rng.normal(0.5, 0.5, shape).astype(np.float32), quats=I.random_squeezed(rng, shape),
                alpha=f(0.01, 0.5), cs=f(0, 1), ct=f(0, 1),
                labels=rng.randint(0, 3, shape).astype(np.uint8) if supervised else None)


def _cut(inp, eigs, num_iter, update, bound=-1.0, alpha=None, scaling=(1, 1, 1), path=0):
    from miccai2016_gb300.continuous_cut_anisotropic_gpu import CmfCutQAnisotropicGpu
    p = CmfCutQAnisotropicGpu.CutParameters()
    p.num_iter, p.update, p.error_bound = num_iter, update, bound
    c = CmfCutQAnisotropicGpu(p)
    c.iteration_path = path
    u = c.execute(inp["img"], inp["quats"], eigs, inp["alpha"] if alpha is None else alpha, inp["cs"], inp["ct"],
                  labels=inp["labels"], scaling=scaling, verbose=False)
    return u, c


@pytest.mark.parametrize("shape", [(1, 16, 32), (2, 17, 33), (3, 29, 60), (9, 30, 61), (5, 42, 88), (40, 15, 89),
                                   (70, 1, 1), (1, 1, 130), (26, 18, 31)])
@pytest.mark.parametrize("eigs", [(1.0, E, E), (1.0, 1.0, 1.0), (E, 1.0, E), (0.3, 0.3, 0.9), (1.0, 0.2, 0.05),
                                  "field"])
@pytest.mark.parametrize("supervised", [False, True])
def test_tiles_match_the_oracle(shape, eigs, supervised):
    inp = _inputs(sum(shape), shape, supervised)
    if eigs == "field":
        eigs = np.random.RandomState(1).uniform(0.01, 2, shape + (3,))
    scaling = (1.5, 0.7, 1.2) if shape[0] % 2 else (1, 1, 1)
    alpha = 0.2 if shape[0] == 9 else None            # a scalar weight once
    kw = dict(num_iter=41, update=7, error_bound=-1.0)
    u, c = _cut(inp, eigs, 41, 7, alpha=alpha, scaling=scaling)
    assert c.last_stats.pair_launches == 20 and c.last_stats.p_launches == 0   # the tile sweeps ran
    a = inp["alpha"] if alpha is None else np.full(shape, alpha, np.float32)
    ru, it, res = O.maxflow_solve(inp["img"], inp["quats"], eigs, a, inp["cs"], inp["ct"], labels=inp["labels"],
                                  scaling=scaling, **kw)
    assert c.last_iterations == it == 41
    assert np.max(np.abs(u - ru)) <= U_TOL
    np.testing.assert_allclose(c.last_residuals, res[:len(c.last_residuals)], rtol=1e-3, atol=1e-7)


@pytest.mark.parametrize("update", [1, 2, 5])
def test_a_stop_gives_the_bits_of_that_many_iterations(update):
    """Bounds between two successive residuals stop the solve after odd and
    even iteration counts."""
    inp = _inputs(5, (20, 37, 45))
    eigs = (1.0, E, E)
    _, full = _cut(inp, eigs, 60, update)
    res = full.last_residuals
    seen = set()
    for k in range(3, 10):
        bound = 0.5 * (res[k] + res[k - 1])
        if not res[k] < bound < res[:k].min():
            continue
        u, c = _cut(inp, eigs, 60, update, bound=float(bound))
        assert c.last_iterations == k * update + 1
        seen.add(c.last_iterations % 2)
        v, _ = _cut(inp, eigs, c.last_iterations, update)
        assert np.array_equal(u.view(np.uint32), v.view(np.uint32)), k
    assert seen == ({1} if update % 2 == 0 else {0, 1})


def test_a_small_workspace_takes_the_two_sweeps():
    import torch
    from miccai2016_gb300 import _native as N
    L = N.lib()
    shape = (12, 20, 40)
    inp = _inputs(6, shape)
    for eigs in ((1.0, E, E), (1.0, 0.2, 0.05)):
        u_tiles, c = _cut(inp, eigs, 30, 10)
        u_two, t = _cut(inp, eigs, 30, 10, path=N.PATH_TWO_SWEEPS)
        assert t.last_stats.pair_launches == 0 and t.last_stats.p_launches == 30
        assert c.last_stats.pair_launches == 15 and c.last_stats.p_launches == 0
        p = N.CutParams(0.2, 0.11, -1.0, 30, 10, (ctypes.c_double * 3)(1, 1, 1))
        nb = L.m16_maxflow_workspace_bytes_min(*shape, ctypes.byref(p))
        assert nb < L.m16_maxflow_workspace_bytes(*shape, ctypes.byref(p))
        d = {k: N.to_device_f32(inp[k]) for k in ("img", "quats", "alpha", "cs", "ct")}
        u = torch.empty(shape, dtype=torch.float32, device="cuda")
        ws = torch.empty(nb, dtype=torch.uint8, device="cuda")
        it = ctypes.c_int32(0)
        args = [N.ptr(d["img"]), N.ptr(d["quats"]), (ctypes.c_double * 3)(*np.sqrt(eigs)), None, N.ptr(d["alpha"]),
                0.0, N.ptr(d["cs"]), N.ptr(d["ct"]), None, *shape, ctypes.byref(p), N.ptr(u), ctypes.byref(it), None,
                0, None, N.ptr(ws)]
        assert L.m16_maxflow_solve(*args, nb - 256, N.stream_ptr()) == N.M16_ERR_WORKSPACE
        assert L.m16_maxflow_solve(*args, nb, N.stream_ptr()) == N.M16_OK
        torch.cuda.synchronize()
        assert np.array_equal(u.cpu().numpy().view(np.uint32), u_two.view(np.uint32))
        assert np.max(np.abs(u_tiles - u_two)) <= U_TOL


@pytest.mark.parametrize("shape", [(1, 1, 3), (5, 17, 33), (64, 64, 64), (90, 120, 140)])   # 1 to 400 blocks
def test_the_last_block_gives_the_residuals(shape):
    """The block that arrives last sums the partials in a fixed order: the
    same bits whatever iterations are checked, solve after solve."""
    inp = _inputs(3, shape)
    u1, c1 = _cut(inp, (1.0, E, E), 29, 1)
    for update in (1, 2, 7):
        u, c = _cut(inp, (1.0, E, E), 29, update)
        assert np.array_equal(u.view(np.uint32), u1.view(np.uint32))
        assert np.array_equal(np.asarray(c.last_residuals), np.asarray(c1.last_residuals)[::update])


def test_the_maximum_of_many_partials():
    """The image's maximum in the last voxel, and a NaN image."""
    shape = (50, 60, 70)
    inp = _inputs(4, shape)
    inp["img"][-1, -1, -1] = 50.0
    u, _ = _cut(inp, (1.0, 1.0, 1.0), 4, 30)
    ru, _, _ = O.maxflow_solve(inp["img"], inp["quats"], (1.0, 1.0, 1.0), inp["alpha"], inp["cs"], inp["ct"],
                               num_iter=4, update=30, error_bound=-1.0)
    assert np.max(np.abs(u - ru)) <= U_TOL
    inp["img"][3, 4, 5] = np.nan
    _, c = _cut(inp, (1.0, 1.0, 1.0), 4, 30)
    assert c.last_iterations == 1 and np.isnan(c.last_residuals[0])   # the reference's check stops at NaN
