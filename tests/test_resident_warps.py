"""The EXACT voxel kernel with a fluence grid, the optional features and any
source (csrc/mcvox_kernel.cuh, mv_min_blocks) keeps 24 warps on an SM."""
import numpy as np
import pytest

import scenarios


@pytest.mark.gpu
@pytest.mark.parametrize('pf', [['Hg', 0.8], ['Gk', 0.8, 0.5], ['Lut'], ['MHg', 0.8, 0.9]])
@pytest.mark.parametrize('method', [0, 1, 2])
def test_threads_of_a_long_run(cuda, lib, method, pf):
    """With many more packets than lanes nearly every resident lane ends one
    (16 warps without the bound)."""
    air = pf[:1] + [0.0] + pf[2:] if len(pf) > 1 else pf
    mc = scenarios.build_mc(dict(
        medium='mcvox', grid=dict(x=[-1e-3, 1e-3, 4], y=[-1e-3, 1e-3, 4], z=[0.0, 1e-3, 4]), layout=dict(kind='uniform'),
        materials=[dict(n=1.0, mua=0.0, mus=0.0, pf=air), dict(n=1.3, mua=1000.0, mus=5e3, pf=pf)],
        source=dict(type='UniformBeam', diameter=5e-4), method=method, rnginit=3,
        detectors=dict(top=dict(type='Total')),
        fluence=dict(x=[-1e-3, 1e-3, 4], y=[-1e-3, 1e-3, 4], z=[0.0, 1e-3, 4], mode='fluence')),
        scheduling='dynamic')
    mc.run(1_000_000)
    sms = cuda.cuda.get_device_properties(0).multi_processor_count
    assert mc.run_report['threads'] >= 0.95 * 24 * 32 * sms
