"""The gradient vector flow on both sides of the rule that chooses its sweeps
(csrc/gvf.cu, gvf_tile_ok), and the edges of the tiles with a response at sizes
that the tile sweeps take (a block has 32 rows and 32 columns, writes 28 of each
and three iterations a pass): against the oracle within the GVF tolerance."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as O


def _run(shape, resp, maxiter, update, callback=None):
    from miccai2016_gb300.gradient_vector_flow import GvfGpu, GvfParameters
    rng = np.random.RandomState(sum(shape))
    v = rng.normal(0, 0.4, shape + (3,)).astype(np.float32)
    r = rng.uniform(0, 1, shape).astype(np.float32) if resp else None
    p = GvfParameters()
    p.mu, p.tol, p.maxiter, p.update, p.callback, p.normalize = 0.2, 0.0, maxiter, update, callback, False
    vs = (1.5, 0.7, 1.2) if shape[0] % 2 else (1.0, 1.0, 1.0)
    obj = GvfGpu(v, p, voxel_size=vs, response=r)
    return obj.execute(), obj, v, r, vs


# blocks of the plain sweep at and above one and two per SM (152), few rows with a short and a long march, single planes
@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(38, 16, 33), (39, 16, 33), (19, 8, 256), (20, 8, 256), (64, 16, 64), (80, 16, 64),
                                   (153, 8, 16), (2000, 3, 34), (40, 9, 700), (40, 10, 700), (40, 11, 700), (40, 12, 700),
                                   (1, 5, 900), (1, 2, 9000), (25, 24, 24)])
@pytest.mark.parametrize("resp", [False, True])
def test_both_sides_of_the_rule(shape, resp):
    for maxiter in (1, 8):
        g, obj, v, r, vs = _run(shape, resp, maxiter, 3)
        ref, _, mags = O.gvf_run(v, 0.2, maxiter, 3, response=r, voxel_size=vs)
        assert np.max(np.abs(g - ref)) <= 1e-4 * max(float(np.max(np.abs(ref))), 1e-6)
        np.testing.assert_allclose(obj.last_mags, mags[:len(obj.last_mags)], rtol=1e-4, atol=1e-9)
    h, _, _, _, _ = _run(shape, resp, 8, 3, callback=lambda f, i, mag: None)   # in pieces, from the same workspace
    assert np.array_equal(g.view(np.uint32), h.view(np.uint32))


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(60, 31, 31), (1, 32, 32), (60, 32, 32), (45, 33, 33), (20, 60, 60), (2, 61, 900),
                                   (3, 89, 300), (200, 89, 3), (20, 88, 61), (150, 33, 2)])
def test_edges_of_the_tiles_with_a_response(shape):
    for maxiter in (1, 2, 3, 4, 5, 13):
        g, obj, v, r, vs = _run(shape, True, maxiter, 4)
        ref, _, mags = O.gvf_run(v, 0.2, maxiter, 4, response=r, voxel_size=vs)
        assert np.max(np.abs(g - ref)) <= 1e-4 * max(float(np.max(np.abs(ref))), 1e-6), maxiter
        np.testing.assert_allclose(obj.last_mags, mags[:len(obj.last_mags)], rtol=1e-4, atol=1e-9)


def test_a_workspace_for_a_response_does_without_one():
    from miccai2016_gb300 import _native as N
    L = N.lib()
    rng = np.random.RandomState(0)
    for k in range(3000):
        d = [int(round(np.exp(rng.uniform(0, np.log(400))))) for _ in range(3)]
        assert L.m16_gvf_workspace_bytes(*d, 1, 16) >= L.m16_gvf_workspace_bytes(*d, 0, 16) >= 36 * d[0] * d[1] * d[2], d
