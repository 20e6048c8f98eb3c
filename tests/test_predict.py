"""Surrogate.predict with inputs and exponential on the device against the
same network driven from the host."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize('m', [1, 7, 129, 4099, (1 << 17) + 3])
def test_predict_equals_host_inputs_and_exponential(cuda, lib, m):
    """Partial row groups, tiles and passes.  Logarithm and exponential of
    host and device are each within an ulp of 2^-53, so profiles agree to a
    few of those; where the ulp of a logarithm falls on a rounding boundary of
    the FP32 feature, its low bf16 part moves by 2^-17 at most, which a
    network with outputs of order 1 over inputs of order 1 cannot turn into
    more than a thousandth."""
    from pyxopto_gb300.surrogate import Mlp, Surrogate, default_weights, features, split_bf16
    rng = np.random.default_rng(m)
    q = (np.exp(rng.uniform(0.0, np.log(1000.0), m)), np.exp(rng.uniform(np.log(500.0), np.log(5000.0), m)),
         rng.uniform(0.6, 0.95, m), rng.uniform(1.33, 1.5, m))
    sur = Surrogate.load(default_weights())
    got = sur.predict(*q)
    assert got.shape == (m, sur.raxis.n) and got.dtype == np.float64
    net = Mlp(sizes=sur.mlp.sizes, batch=(m + 7) // 8 * 8)
    net.load_state(*sur.mlp.state())
    x = np.zeros(((m + 7) // 8 * 8, 16), np.float32)
    x[:m] = features(*q)
    z = net.forward(split_bf16(x), store=False)[:m, :sur.raxis.n].cpu().numpy().astype(np.float64)
    want = np.exp(sur.mu[None, :] + sur.scale * z)
    err = np.max(np.abs(got / want - 1.0), axis=1)
    assert np.mean(err > 1e-14) <= 1e-3 and np.max(err) < 1e-3
    # scalars broadcast over the queries, as in features()
    one = sur.predict(q[0], q[1], 0.8, 1.4)
    assert np.array_equal(one, sur.predict(q[0], q[1], np.full(m, 0.8), np.full(m, 1.4)))


def test_predict_refuses_no_queries(lib):
    from pyxopto_gb300.surrogate import Surrogate
    with pytest.raises(ValueError):
        sur = Surrogate()
        sur.mlp = type('Net', (), {'w': [0]})()
        sur.predict([], [], [], [])
