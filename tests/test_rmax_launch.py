"""Packets launched farther than rmax from the source position
(csrc/mcml_kernel.cuh): the first step moves them, crosses the boundary that
it reaches and deposits in the detector there before rmax ends them."""
import numpy as np
import pytest

import scenarios

SOURCES = {
    'UniformBeam': dict(type='UniformBeam', diameter=4e-3),
    'GaussianBeam': dict(type='GaussianBeam', sigma=1.5e-3, clip=3.0),
    'UniformRectangular': dict(type='UniformRectangular', width=4e-3, height=3e-3, na=0.2),
    'IsotropicPoint': dict(type='IsotropicPoint', position=(0.0, 0.0, -1e-3)),
}


def _spec(source, fluence):
    air = dict(d=0.0, n=1.0, mua=0.0, mus=0.0, pf=['Hg', 0.0])
    s = dict(medium='mcml', layers=[air, dict(d=1e-4, n=1.0, mua=10.0, mus=1e3, pf=['Hg', 0.5]), air],
             source=SOURCES[source], rmax=1.5e-3, rnginit=5,
             detectors=dict(top=dict(type='Total'), bottom=dict(type='Radial', axis=[0.0, 4e-3, 20])))
    if fluence:
        s['fluence'] = dict(x=[-2e-3, 2e-3, 9], y=[-2e-3, 2e-3, 7], z=[0.0, 1e-4, 3], mode='deposition')
    return s


@pytest.mark.gpu
@pytest.mark.parametrize('fluence', [False, True])
@pytest.mark.parametrize('source', sorted(SOURCES))
def test_launch_beyond_rmax_bit_identical_to_oracle(cuda, lib, oracle, source, fluence):
    mc = scenarios.build_mc(_spec(source, fluence), scheduling='dynamic')
    ref = oracle.run(mc, 4000, 0, oracle.PORTABLE, nthreads=8)
    mc.run(4000)
    got = oracle.tallies(mc, mc._dev['accu'].cpu().numpy().view(np.uint64))
    for k in got:
        assert np.array_equal(got[k], ref[k]), k
    assert mc.run_report['steps'] == ref['steps']


@pytest.mark.gpu
@pytest.mark.parametrize('source', sorted(SOURCES))
def test_launch_beyond_rmax_fast(cuda, lib, oracle, source):
    """FAST math runs the packets of the EXACT oracle; only one whose path a
    rounding changes differs, so the collected weights differ by far less
    than 5 sigma of two independent runs, 5 sqrt(2 n / 4)."""
    n = 20000
    mc = scenarios.build_mc(_spec(source, False), fast=True, scheduling='dynamic')
    ref = oracle.run(mc, n, 0, oracle.PORTABLE, nthreads=8)
    dets = mc.run(n)[2]
    for slot in ('top', 'bottom'):
        got = getattr(dets, slot).raw.sum()
        assert abs(got - ref[slot].sum() / 8388607.0) <= 5.0 * (n / 2.0) ** 0.5, slot
