"""Float tables that the transport kernels stage in shared memory, up to
24,576 floats: the table and the kernel's own tables together pass the 48 KB
that need no opt-in at sizes of their own per kernel."""
import importlib

import numpy as np
import pytest

import scenarios


def _mc(medium, scheduling, floats, trace):
    """A simulator whose phase functions take the given number of floats."""
    m = importlib.import_module('pyxopto_gb300.{}.mc'.format(medium))

    def pf(n):
        return m.mcpf.Lut(*scenarios.lut_table(n))

    opts = [m.mcoptions.McScheduling(scheduling)]
    dets = m.mcdetector.Detectors(top=m.mcdetector.Total())
    tr = m.mctrace.Trace(maxlen=8) if trace else None
    if medium == 'mcml':
        L = m.mclayer.Layer
        layers = m.mclayer.Layers([L(d=0.0, n=1.0, mua=0.0, mus=0.0, pf=pf(2)),
                                   L(d=1e-3, n=1.3, mua=100.0, mus=1e4, pf=pf(floats - 4)),
                                   L(d=0.0, n=1.0, mua=0.0, mus=0.0, pf=pf(2))])
        return m.Mc(layers, m.mcsource.Line(), dets, trace=tr, options=opts, rnginit=3)
    A = m.mcdetector.Axis
    vox = m.mcgeometry.Voxels(A(-1e-3, 1e-3, 4), A(-1e-3, 1e-3, 4), A(0.0, 1e-3, 4))
    vox.material[...] = 1
    M = m.mcmaterial.Material
    mats = [M(n=1.0, mua=0.0, mus=0.0, pf=pf(2)), M(n=1.3, mua=100.0, mus=1e4, pf=pf(floats - 2))]
    return m.Mc(vox, mats, m.mcsource.Line(), dets, trace=tr, options=opts, rnginit=3)


@pytest.mark.gpu
@pytest.mark.parametrize('trace', [False, True])
@pytest.mark.parametrize('scheduling', ['static', 'dynamic'])
@pytest.mark.parametrize('medium', ['mcml', 'mcvox'])
@pytest.mark.parametrize('floats', [7400, 7800, 10300, 10700, 12280, 12288, 12292, 24576, 24577])
def test_table_sizes_bit_identical_to_oracle(cuda, lib, oracle, medium, scheduling, trace, floats):
    n = 300
    mc = _mc(medium, scheduling, floats, trace)
    ref = oracle.run(mc, n, 64, oracle.PORTABLE)
    mc.run(n, maxthreads=64)
    assert mc._lut_array().size == floats
    got = oracle.tallies(mc, mc._dev['accu'].cpu().numpy().view(np.uint64))
    assert np.array_equal(got['top'], ref['top'])
    assert mc.run_report['steps'] == ref['steps']
