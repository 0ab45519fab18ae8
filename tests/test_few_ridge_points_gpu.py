"""The nearest-ridge sign flip for few ridge points (csrc/directions.cu,
dr_adjust_few_kernel: up to 16384 points and one per 32 voxels) against the
brute-force kernel, bit for bit: volumes that end inside a block of 8 x 8 x 8,
lists that end inside a round of 256 points, ties, points outside the volume,
both sides of the rule."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _flip(vecs, coords, rdirs, scaling, indexed):
    import torch
    from miccai2016_gb300 import _native as N
    L = N.lib()
    d = torch.from_numpy(vecs).cuda()
    c = torch.from_numpy(np.ascontiguousarray(coords, np.uint16).view(np.int16)).cuda()
    r = torch.from_numpy(rdirs).cuda()
    sc = (ctypes.c_double * 3)(*scaling)
    if indexed:
        ws = N.workspace(L.m16_adjust_nonridge_signs_workspace_bytes(*vecs.shape[:3], len(coords)))
        st = L.m16_adjust_nonridge_signs_indexed(N.ptr(d), *vecs.shape[:3], N.ptr(c), N.ptr(r), len(coords), sc,
                                                 N.ptr(ws), ws.numel(), N.stream_ptr())
    else:
        st = L.m16_adjust_nonridge_signs(N.ptr(d), *vecs.shape[:3], N.ptr(c), N.ptr(r), len(coords), sc,
                                         N.stream_ptr())
    N.check("sign flip", st)
    return d.cpu().numpy()


@pytest.mark.parametrize("shape,points", [((1, 1, 32), 1), ((7, 8, 9), 2), ((8, 8, 8), 16), ((8, 8, 8), 17),
                                          ((17, 9, 64), 255), ((17, 9, 64), 306), ((17, 9, 64), 307),
                                          ((33, 31, 40), 256), ((33, 31, 40), 257), ((33, 31, 40), 1200),
                                          ((90, 80, 75), 16384), ((90, 80, 75), 16385)])
@pytest.mark.parametrize("scaling", [(1, 1, 1), (1.5, 0.7, 1.2), (1e-3, 40.0, 1.0)])
@pytest.mark.parametrize("lattice", [1, 4])   # 4: a coarse lattice, most voxels with ties
def test_equals_brute_force(shape, points, scaling, lattice):
    rng = np.random.RandomState(points + lattice)
    coords = rng.randint(0, np.array(shape) + (0, 0, 5), (points, 3)) // lattice * lattice
    vecs = rng.normal(size=shape + (3,)).astype(np.float32)
    rdirs = rng.normal(size=(points, 3)).astype(np.float32)
    a = _flip(vecs, coords, rdirs, scaling, True)
    b = _flip(vecs, coords, rdirs, scaling, False)
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32))


def test_points_in_one_corner_of_a_long_volume():
    """Every point is a candidate of the far blocks' bound only by its rounding."""
    shape = (3, 5, 3000)
    rng = np.random.RandomState(1)
    coords = rng.randint(0, (3, 5, 6), (300, 3))
    vecs = rng.normal(size=shape + (3,)).astype(np.float32)
    rdirs = rng.normal(size=(300, 3)).astype(np.float32)
    for scaling in ((1, 1, 1), (0.3333, 0.3333, 0.3333)):
        a = _flip(vecs, coords, rdirs, scaling, True)
        assert np.array_equal(a.view(np.uint32), _flip(vecs, coords, rdirs, scaling, False).view(np.uint32))
