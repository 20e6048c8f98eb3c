"""The one-call training step (csrc/mlp_step.cuh) against the separate
kernels: the same products, roundings and sums over rows."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize('mode', [0, 1])
@pytest.mark.parametrize('m', [8, 40, 136, 1000, 4096, 9000])
@pytest.mark.parametrize('sizes', [(4, 256, 256, 256, 30), (4, 48, 30), (4, 64, 144, 17)])
def test_fused_step_equals_separate_kernels(cuda, sizes, m, mode):
    """Rows beyond the last tile, chunk and slice, one to eight accumulators
    per weight-gradient block, tile edges in the widths: every tensor is equal
    after each of three steps.  Only the loss is summed in another order: of
    up to 32 m terms of one sign, each rounding at most 2^-24 of the sum."""
    from pyxopto_gb300.surrogate import Mlp
    torch = cuda
    nv = sizes[-1]
    rng = np.random.default_rng(m + mode)
    a, b = (Mlp(sizes=sizes, seed=3, batch=m) for _ in range(2))
    x = torch.zeros((m, 16), dtype=torch.bfloat16, device='cuda')
    x[:, :8] = torch.from_numpy(rng.uniform(-1, 1, (m, 8)).astype(np.float32)).cuda()
    t = torch.from_numpy(np.exp(0.5 * rng.normal(0, 1, (m, 32))).astype(np.float32)).cuda()
    b._one_call = lambda *args: False
    for step in range(3):
        la = a.train_step(x, t, nv, 1e-3, mode=mode, scale=0.7).double().sum()
        lb = b.train_step(x, t, nv, 1e-3, mode=mode, scale=0.7).double().sum()
        assert abs(la - lb) <= 2.0 ** -24 * max(8.0, (32 * m) ** 0.5) * lb
        for name in ('pre', 'dpre', 'dw', 'db', 'w', 'b', 'wb', 'wt', 'm', 'v', 'bb', 'mb', 'vb'):
            for u, v in zip(getattr(a, name), getattr(b, name)):
                assert torch.equal(u, v), (step, name)
    assert torch.equal(a.h[0], b.h[0]) and a.step_count == b.step_count == 3
