"""Rows of more than 2^29 voxels: a tensor copy's coordinate along x counts four
floats a voxel and is a 32-bit number, so these volumes take the sweeps without
tensor copies.  Their workspace sizes say so (nothing of this size is run)."""
import ctypes

import pytest

LONGEST = (2 ** 31 - 1) // 4 - 3   # padded, times four, still below 2^31


@pytest.fixture(scope="module")
def lib():
    from miccai2016_gb300 import _native
    return _native.lib()


@pytest.mark.parametrize("d2", [LONGEST, LONGEST + 1, 2 ** 29, 600_000_000, 2 ** 31 - 4, 2 ** 31 - 1])
def test_long_rows_take_the_two_sweeps(lib, d2):
    from miccai2016_gb300 import _native as N
    p = N.CutParams(0.2, 0.11, 1e-4, 100, 10, (ctypes.c_double * 3)(1, 1, 1))
    whole = lib.m16_maxflow_workspace_bytes(1, 1, d2, ctypes.byref(p))
    least = lib.m16_maxflow_workspace_bytes_min(1, 1, d2, ctypes.byref(p))
    assert 36 * d2 <= least <= 37 * d2
    if d2 <= LONGEST:
        assert 4 * (d2 + 3) < 2 ** 31 and whole >= 88 * d2
    else:
        assert whole == least
    # a served request: 72 bytes a voxel with the tile sweeps, 68 without
    per_voxel = lib.m16_server_request_bytes(1, 1, d2, 0) / d2
    assert per_voxel >= 72 if d2 <= LONGEST else 68 <= per_voxel < 69
    # a field: the padded copies need no less than the plain ones
    assert lib.m16_gvf_workspace_bytes(1, 1, d2, 0, 8) >= 36 * d2
