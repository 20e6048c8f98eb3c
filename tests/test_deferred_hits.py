"""Layered steps whose boundary hits are processed together after several
steps of the warp (csrc/mcml_kernel.cuh): bit-identical to the oracle."""
import numpy as np
import pytest

import scenarios

INF = float('inf')


def _spec(pf, layers, fluence, rmax):
    air = dict(d=0.0, n=1.0, mua=0.0, mus=0.0, pf=pf)
    s = dict(medium='mcml', layers=[air] + [dict(l, pf=[pf[0]] + l['pf']) for l in layers] + [air],
             source=dict(type='Line'),
             detectors=dict(top=dict(type='Radial', axis=[0.0, 2e-3, 20]), bottom=dict(type='Total'),
                            specular=dict(type='Total')), rnginit=11)
    if fluence:
        s['fluence'] = dict(x=[-1e-3, 1e-3, 9], y=[-1e-3, 1e-3, 7], z=[0.0, 2e-3, 11], mode='deposition')
    if rmax:
        s['rmax'] = rmax
    return s


@pytest.mark.gpu
@pytest.mark.parametrize('fluence', [False, True])
@pytest.mark.parametrize('rmax', [None, 1e-3])
@pytest.mark.parametrize('pf', ['Hg', 'Gk'])
@pytest.mark.parametrize('layers', ['empty layer', 'thin layers', 'mismatch', 'half space'])
def test_hits_bit_identical_to_oracle(cuda, lib, oracle, layers, pf, rmax, fluence):
    """A layer of no thickness (a path that reaches it ends inside after
    all), layers thinner than a free path (a hit at nearly every step),
    refractive-index steps and total reflection, and a semi-infinite one."""
    p = [0.8] if pf == 'Hg' else [0.8, 0.5]
    iso = [0.0] if pf == 'Hg' else [0.0, 0.5]
    stack = {
        'empty layer': [dict(d=4e-4, n=1.4, mua=100.0, mus=1e4, pf=p), dict(d=0.0, n=1.4, mua=50.0, mus=2e4, pf=p),
                        dict(d=6e-4, n=1.4, mua=10.0, mus=1e4, pf=iso)],
        'thin layers': [dict(d=1e-7, n=1.4, mua=100.0, mus=1e4, pf=p), dict(d=3e-6, n=1.35, mua=0.0, mus=1e4, pf=p),
                        dict(d=2e-5, n=1.5, mua=300.0, mus=0.0, pf=p), dict(d=1e-3, n=1.33, mua=20.0, mus=9e3, pf=p)],
        'mismatch': [dict(d=3e-4, n=1.8, mua=50.0, mus=1.5e4, pf=p), dict(d=5e-4, n=1.1, mua=30.0, mus=8e3, pf=iso)],
        'half space': [dict(d=INF, n=1.37, mua=30.0, mus=1.2e4, pf=p)],
    }[layers]
    mc = scenarios.build_mc(_spec([pf] + iso, stack, fluence, rmax), scheduling='dynamic')
    ref = oracle.run(mc, 3000, 0, oracle.PORTABLE, nthreads=8)
    mc.run(3000)
    got = oracle.tallies(mc, mc._dev['accu'].cpu().numpy().view(np.uint64))
    for k in got:
        assert np.array_equal(got[k], ref[k]), k
    assert mc.run_report['steps'] == ref['steps']
