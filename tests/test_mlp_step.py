"""The one-call training step (csrc/mlp_step.cuh) against the separate
kernels: the same products and roundings, other orders of the FP32 sums over
rows."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize('mode', [0, 1])
@pytest.mark.parametrize('m', [8, 136, 1000, 4096, 9000])
@pytest.mark.parametrize('sizes', [(4, 256, 256, 256, 30), (4, 48, 30), (4, 64, 144, 17)])
def test_fused_step_equals_separate_kernels(cuda, sizes, m, mode):
    """Rows beyond the last tile and slice, one to four accumulators per
    weight-gradient block, tile edges in the widths.  A sum of up to m terms
    in another order moves by at most m rounding errors of its largest
    partial sum; 2^-24 sqrt(m) relative to the tensor's norm covers the
    gradients with room (FP32 accumulation of bf16 products)."""
    from pyxopto_gb300.surrogate import Mlp
    torch = cuda
    nv = sizes[-1]
    rng = np.random.default_rng(m + mode)
    a, b = (Mlp(sizes=sizes, seed=3, batch=m) for _ in range(2))
    x = torch.zeros((m, 16), dtype=torch.bfloat16, device='cuda')
    x[:, :8] = torch.from_numpy(rng.uniform(-1, 1, (m, 8)).astype(np.float32)).cuda()
    t = torch.from_numpy(np.exp(0.5 * rng.normal(0, 1, (m, 32))).astype(np.float32)).cuda()
    b._one_call = lambda *args: False
    la = a.train_step(x, t, nv, 1e-3, mode=mode, scale=0.7).double()
    lb = b.train_step(x, t, nv, 1e-3, mode=mode, scale=0.7).double()
    tol = 2.0 ** -24 * max(4.0, m ** 0.5) * 4
    assert (la - lb).norm() <= tol * lb.norm()
    for name in ('dw', 'db'):
        for u, v in zip(getattr(a, name), getattr(b, name)):
            assert (u.double() - v.double()).norm() <= tol * v.double().norm(), name
    for u, v in zip(a.pre, b.pre):
        assert torch.equal(u, v)
    for u, v in zip(a.dpre, b.dpre):
        assert torch.equal(u, v)
    assert torch.equal(a.h[0], b.h[0]) and a.step_count == b.step_count == 1
    # AdamW from the same gradients: the update equals the separate kernel's
    c = Mlp(sizes=sizes, seed=3, batch=m)
    for u, v in zip(c.dw + c.db, a.dw + a.db):
        u.copy_(v)
    c.adamw(lr=1e-3)
    for name in ('w', 'b', 'wb', 'wt', 'm', 'v', 'bb', 'mb', 'vb'):
        for u, v in zip(getattr(a, name), getattr(c, name)):
            assert torch.equal(u, v), name
