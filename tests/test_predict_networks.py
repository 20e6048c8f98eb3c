"""Surrogate.predict of networks and normalisations that the one-call path
does not take."""
import numpy as np
import pytest


def _surrogate(sizes, seed=2, batch=264):
    from pyxopto_gb300.surrogate import Mlp, Surrogate
    sur = Surrogate()
    sur.mlp = Mlp(sizes=sizes, seed=seed, batch=batch)
    rng = np.random.default_rng(seed)
    sur.mu, sur.scale = rng.normal(0.0, 1.0, 30), 0.7
    return sur


def _queries(m):
    rng = np.random.default_rng(m)
    return (np.exp(rng.uniform(0.0, np.log(1000.0), m)), np.exp(rng.uniform(np.log(500.0), np.log(5000.0), m)),
            rng.uniform(0.6, 0.95, m), rng.uniform(1.33, 1.5, m))


@pytest.mark.gpu
@pytest.mark.parametrize('hidden', [7, 8, 11])
@pytest.mark.parametrize('m', [1, 263, 529])
def test_deep_networks(cuda, lib, hidden, m):
    """Around the eight layers of the one call, over more queries than the
    network's batch, against the network driven from here: equal but for an
    ulp of logarithm and exponential, which can move the low bf16 part of an
    input by 2^-17 of it."""
    from pyxopto_gb300.surrogate import Mlp, features, split_bf16
    sizes = (4,) + (32,) * hidden + (30,)
    sur = _surrogate(sizes)
    q = _queries(m)
    got = sur.predict(*q)
    assert got.shape == (m, 30) and got.dtype == np.float64
    net = Mlp(sizes=sizes, batch=(m + 7) // 8 * 8)
    net.load_state(*sur.mlp.state())
    x = np.zeros((net.batch, 16), np.float32)
    x[:m] = features(*q)
    z = net.forward(split_bf16(x))[:m, :30].cpu().numpy().astype(np.float64)
    assert np.max(np.abs(got / np.exp(sur.mu + sur.scale * z) - 1.0)) < 1e-3


@pytest.mark.gpu
def test_normalisation_of_another_length_is_refused(cuda, lib):
    sur = _surrogate((4, 64, 30))
    sur.mu = sur.mu[:20]
    with pytest.raises(ValueError):
        sur.predict(*_queries(9))


@pytest.mark.gpu
def test_normalisation_per_bin(cuda, lib):
    sur = _surrogate((4, 64, 30))
    q = _queries(9)
    one = sur.predict(*q)
    sur.scale = np.full(30, sur.scale)
    assert np.max(np.abs(sur.predict(*q) / one - 1.0)) < 1e-3
