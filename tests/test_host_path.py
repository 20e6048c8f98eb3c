"""The run cycle around the kernels: tallies scaled on the device, and the
voxel grid kept between runs by its content."""
import numpy as np
import pytest

import scenarios


@pytest.mark.gpu
@pytest.mark.parametrize('n', [1, 255, 257, 100_003])
def test_scaled_tallies_equal_numpy(cuda, lib, n):
    from pyxopto_gb300 import _lib
    rng = np.random.default_rng(n)
    raw = rng.integers(0, 2 ** 63, n, dtype=np.uint64) >> rng.integers(0, 63, n, dtype=np.uint64)
    mc = scenarios.build_mc('c1_line_hg_radial')
    dev = cuda.from_numpy(raw.view(np.int64)).cuda()
    assert np.array_equal(mc._scaled(cuda, dev, 1.0 / 8388607), raw * (1.0 / 8388607))
    big = np.full(n, 2 ** 64 - 1, np.uint64)
    assert np.array_equal(mc._scaled(cuda, cuda.from_numpy(big.view(np.int64)).cuda(), 0.3), big * 0.3)
    assert _lib.load().mcgb_scale_u64(None, 0, 1.0, None, None) == 0


@pytest.mark.gpu
def test_changed_voxels_are_seen(cuda, lib, oracle):
    """A voxel changed in place, and changed back, between runs of one
    simulator; a material index beyond the list is refused every time."""
    def fresh(change, run):
        m = scenarios.build_mc('c3_vox_cylinder', scheduling='dynamic', fast=True)
        change(m)
        m._packets_total = run * 4000
        return m.run(4000)[1].raw

    mc = scenarios.build_mc('c3_vox_cylinder', scheduling='dynamic', fast=True)
    old = mc.voxels.material[5, 4, 3].copy()

    def one(m):
        m.voxels.material[2:6, 3:6, 3:6] = 2

    a = mc.run(4000)[1].raw
    keep = mc.voxels.material.copy()
    one(mc)
    b = mc.run(4000)[1].raw
    mc.voxels.material[...] = keep
    c = mc.run(4000)[1].raw
    assert np.array_equal(a, fresh(lambda m: None, 0))
    assert np.array_equal(b, fresh(one, 1)) and not np.array_equal(b, fresh(lambda m: None, 1))
    assert np.array_equal(c, fresh(lambda m: None, 2))
    mc.voxels.material[5, 4, 3] = 200
    for _ in range(2):
        with pytest.raises(ValueError):
            mc.run(10)
    mc.voxels.material[5, 4, 3] = old
    mc.run(10)
