"""The sampling-volume kernel over its launch shapes: one to 32 packets per
warp and more packets than lanes, traces of one and two events, and walks
along the axes, bit-identical to the oracle."""
import numpy as np
import pytest

from test_gpu_parity import _sv_expected


@pytest.mark.gpu
@pytest.mark.parametrize('n,maxlen', [(1, 40), (1823, 40), (1825, 3), (60_001, 12), (200_000, 2), (3000, 1)])
def test_shapes_bit_identical_to_oracle(cuda, lib, oracle, n, maxlen):
    from pyxopto_gb300.mcml import mc
    layers = mc.mclayer.Layers([
        mc.mclayer.Layer(d=0.0, n=1.0, mua=0.0, mus=0.0, pf=mc.mcpf.Hg(0.0)),
        mc.mclayer.Layer(d=2e-3, n=1.4, mua=100.0, mus=1e4, pf=mc.mcpf.Hg(0.85)),
        mc.mclayer.Layer(d=0.0, n=1.0, mua=0.0, mus=0.0, pf=mc.mcpf.Hg(0.0))])
    # every event of a Line source's first path lies on the z axis: two
    # direction components are zero there
    sim = mc.Mc(layers, mc.mcsource.Line(), trace=mc.mctrace.Trace(maxlen=maxlen),
                options=[mc.mcoptions.McUseNativeMath(True)], rnginit=5)
    trace, _, _ = sim.run(n)
    A = mc.mcsv.Axis
    sv = mc.mcsv.SamplingVolume(A(-1e-3, 1e-3, 31), A(-1e-3, 1e-3, 20), A(0.0, 2e-3, 47))
    sim.sampling_volume(trace, sv)
    data, weight = _sv_expected(oracle, sim, sv, trace)
    assert np.array_equal(sv.data, data) and sv.weight == weight
