"""mcgb_voxel_radius over grid shapes: lines shorter and longer than a block's
shared memory, partial tiles, flat grids; against scipy's chessboard distance
transform."""
import ctypes as C

import numpy as np
import pytest


def _distance(mat, cap):
    from scipy import ndimage
    low, high = (f(mat, size=3, mode='nearest') for f in (ndimage.minimum_filter, ndimage.maximum_filter))
    inside = low == high
    for axis in range(3):
        edge = [slice(None)] * 3
        for edge[axis] in (0, -1):
            inside[tuple(edge)] = False
    return np.minimum(ndimage.distance_transform_cdt(inside, metric='chessboard'), cap)


@pytest.mark.gpu
@pytest.mark.parametrize('shape', [(1, 1, 1), (200, 3, 5), (70, 65, 130), (129, 128, 127), (3, 900, 40),
                                   (5, 6145, 4), (50_000, 3, 3), (64, 33, 768)])
@pytest.mark.parametrize('cap', [1, 31, 64])
def test_radius_equals_chessboard_distance(cuda, lib, shape, cap):
    from pyxopto_gb300 import _lib
    nx, ny, nz = shape
    rng = np.random.default_rng(nx)
    mat = np.ones((nz, ny, nx), np.uint8)
    for _ in range(6):
        at = [int(rng.integers(0, n)) for n in (nz, ny, nx)]
        mat[at[0]:at[0] + 2, at[1]:at[1] + 3, at[2]:at[2] + 1] = int(rng.integers(2, 5))
    dev = cuda.from_numpy(mat.reshape(-1)).cuda()
    rad = cuda.full_like(dev, 77)
    _lib.check(lib.mcgb_voxel_radius(C.c_void_p(dev.data_ptr()), (C.c_int32 * 3)(nx, ny, nz),
                                     C.c_void_p(rad.data_ptr()), cap, None))
    assert np.array_equal(rad.cpu().numpy().reshape(mat.shape), _distance(mat, cap))
