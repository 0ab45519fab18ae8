"""The GVF sweeps of several iterations per pass (csrc/gvf_tile.cuh): volume
sizes at the blocks' edges, iteration counts that leave a remainder, runs in
pieces, and stops inside a sweep -- each against the oracle within the GVF
tolerance (1e-4 of the largest magnitude) or bit for bit against a run of the
same number of iterations."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden"))

from oracle import oracle as O  # noqa: E402

pytestmark = pytest.mark.gpu


def _gvf(v, maxiter, update, tol=0.0, response=None, callback=None, voxel_size=None):
    from miccai2016_gb300.gradient_vector_flow import GvfGpu, GvfParameters
    p = GvfParameters()
    p.mu, p.maxiter, p.update, p.tol, p.normalize, p.callback = 0.2, maxiter, update, tol, False, callback
    obj = GvfGpu(v, p, voxel_size=voxel_size, response=response)
    return obj.execute(), obj


def _field(seed, shape):
    return np.random.RandomState(seed).normal(0, 0.4, shape + (3,)).astype(np.float32)


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 1, 33), (1, 24, 32), (3, 25, 31), (4, 23, 63), (5, 46, 62),
                                   (6, 47, 64), (40, 3, 5), (9, 70, 95), (33, 24, 2)])
@pytest.mark.parametrize("with_response", [False, True])
def test_edges_match_the_oracle(shape, with_response):
    v = _field(sum(shape), shape)
    r = np.random.RandomState(3).uniform(0, 1, shape).astype(np.float32) if with_response else None
    vs = (1.2, 0.8, 1.0) if shape[0] % 2 else None
    for maxiter in (1, 2, 7, 12):
        g, obj = _gvf(v, maxiter, 5, response=r, voxel_size=vs)
        ref, _, mags = O.gvf_run(v, 0.2, maxiter, 5, response=r, voxel_size=vs)
        assert np.max(np.abs(g - ref)) <= 1e-4 * max(float(np.max(np.abs(ref))), 1e-6), maxiter
        np.testing.assert_allclose(obj.last_mags, mags[:len(obj.last_mags)], rtol=1e-4, atol=1e-9)


@pytest.mark.parametrize("update", [1, 2, 3, 4])
def test_a_stop_inside_a_sweep_gives_the_bits_of_that_many_iterations(update):
    """A nearly constant field: g approaches it and |delta| falls from check to
    check, so a bound between two checks stops at the later one."""
    v = (np.float32([0.5, 0.4, 0.3]) + 0.1 * _field(9, (20, 41, 50))).astype(np.float32)
    _, full = _gvf(v, 20, update)
    m = full.last_mags
    assert np.all(np.diff(m) < 0)
    for k in range(1, len(m)):
        g, obj = _gvf(v, 20, update, tol=float(0.5 * (m[k] + m[k - 1])))
        assert obj.last_iterations == k * update + 1
        h, _ = _gvf(v, obj.last_iterations, update)
        assert np.array_equal(g.view(np.uint32), h.view(np.uint32)), k


def test_pieces_give_the_bits_of_the_whole():
    v = _field(11, (13, 30, 45))
    seen = []
    g, obj = _gvf(v, 23, 4, callback=lambda f, i, mag: seen.append((i, mag)))
    h, whole = _gvf(v, 23, 4)
    assert [i for i, _ in seen] == [0, 4, 8, 12, 16, 20]
    assert np.array_equal(g.view(np.uint32), h.view(np.uint32))
    assert obj.last_iterations == whole.last_iterations == 23


# with a response a block has 32 rows and three iterations a pass
@pytest.mark.parametrize("shape", [(3, 31, 31), (1, 32, 32), (7, 33, 33), (5, 60, 60), (2, 61, 61), (70, 89, 3)])
def test_edges_with_a_response(shape):
    v = _field(sum(shape), shape)
    r = np.random.RandomState(3).uniform(0, 1, shape).astype(np.float32)
    for maxiter in (1, 2, 3, 4, 5, 13):
        g, obj = _gvf(v, maxiter, 4, response=r)
        ref, _, mags = O.gvf_run(v, 0.2, maxiter, 4, response=r)
        assert np.max(np.abs(g - ref)) <= 1e-4 * max(float(np.max(np.abs(ref))), 1e-6), maxiter
        np.testing.assert_allclose(obj.last_mags, mags[:len(obj.last_mags)], rtol=1e-4, atol=1e-9)


@pytest.mark.parametrize("update", [1, 2, 3, 4])
def test_stops_and_pieces_with_a_response(update):
    """The response that is taken without one, |v|^2, given as a field."""
    v = (np.float32([0.5, 0.4, 0.3]) + 0.1 * _field(9, (20, 41, 50))).astype(np.float32)
    r = np.sum(v.astype(np.float64) ** 2, -1).astype(np.float32)
    whole, full = _gvf(v, 20, update, response=r)
    m = full.last_mags
    assert np.all(np.diff(m) < 0)
    for k in range(1, len(m)):
        g, obj = _gvf(v, 20, update, tol=float(0.5 * (m[k] + m[k - 1])), response=r)
        assert obj.last_iterations == k * update + 1
        h, _ = _gvf(v, obj.last_iterations, update, response=r)
        assert np.array_equal(g.view(np.uint32), h.view(np.uint32)), k
    p, _ = _gvf(v, 20, update, response=r, callback=lambda f, i, mag: None)
    assert np.array_equal(p.view(np.uint32), whole.view(np.uint32))
