"""The scratch of the one-call training step (csrc/mlp_step.cuh): sized once
for the largest batch, used by every smaller one."""
import ctypes as C

import numpy as np
import pytest

from pyxopto_gb300 import _abi

NETS = [(16, 256, 256, 256, 32), (16, 48, 32), (16, 64, 144, 32), (16, 512, 512, 32), (16, 1024, 32)]


def _tensors(pads):
    tab = (_abi.McgbAdamwTensor * (2 * (len(pads) - 1)))()
    for i in range(len(pads) - 1):
        tab[2 * i].rows, tab[2 * i].cols = pads[i + 1], pads[i]
        tab[2 * i + 1].rows, tab[2 * i + 1].cols = 1, pads[i + 1]
    return tab


def _used(lib, pads, m):
    """Floats that a step of m rows writes: loss sums, and per layer at most
    eight partial weight gradients, by slices of whole chunks of 64 rows that
    cover 152 SMs twice, and a bias sum per 64 rows."""
    n = ((m + 31) // 32 * 2 + 3) // 4 * 4
    for k, r in zip(pads, pads[1:]):
        tiles = ((r + 127) // 128) * ((k + 63) // 64)
        fine = max(1, min((2 * 152 + tiles - 1) // tiles, m // 64, 64))
        rows = (-(-m // fine) + 63) // 64 * 64
        n += min(-(-m // rows), 8) * r * k + (m + 63) // 64 * r
    return n


@pytest.mark.parametrize('pads', NETS)
def test_scratch_of_a_batch_serves_every_smaller_one(lib, pads):
    tab = _tensors(pads)
    most = 0
    for m in range(8, 6000, 8):
        n = int(lib.mcgb_mlp_train_scratch(tab, len(pads) - 1, m))
        most = max(most, _used(lib, pads, m))
        assert n >= most, m


def test_step_refuses_a_small_scratch(lib, cuda_absent):
    """Refused before anything is launched (the pointers are not memory)."""
    from pyxopto_gb300 import _lib
    pads = NETS[0]
    tab = _tensors(pads)
    s = _abi.McgbMlpStep()
    s.tensors, s.layers = tab, len(pads) - 1
    for t in tab:
        t.w = t.w_bf16 = t.wt_bf16 = t.grad = t.m = t.v = 4096
    for i in range(s.layers):
        s.h[i] = s.pre[i] = s.dpre[i] = 4096
    s.x = s.target = s.loss = s.scratch = 4096
    s.m, s.nv, s.step = 448, 30, 1
    s.scratch_size = int(lib.mcgb_mlp_train_scratch(tab, s.layers, 448)) - 1
    assert lib.mcgb_mlp_train_step(C.byref(s), None) == _abi.E_SIZE
    with pytest.raises(_lib.McgbError):
        _lib.check(lib.mcgb_mlp_train_step(C.byref(s), None))


@pytest.fixture
def cuda_absent():
    import torch
    if torch.cuda.is_available():
        pytest.skip('made-up pointers: only where nothing can be launched')


@pytest.mark.gpu
@pytest.mark.parametrize('batch,steps', [(504, (448, 192, 504)), (264, (256, 8)), (520, (512,))])
def test_smaller_steps_equal_separate_kernels(cuda, batch, steps):
    """Batches whose own slices are fewer than those of a smaller step."""
    from pyxopto_gb300.surrogate import Mlp
    torch = cuda
    rng = np.random.default_rng(batch)
    a, b = (Mlp(seed=3, batch=batch) for _ in range(2))
    b._one_call = lambda *args: False
    for m in steps:
        x = torch.zeros((m, 16), dtype=torch.bfloat16, device='cuda')
        x[:, :8] = torch.from_numpy(rng.uniform(-1, 1, (m, 8)).astype(np.float32)).cuda()
        t = torch.from_numpy(np.exp(0.5 * rng.normal(0, 1, (m, 32))).astype(np.float32)).cuda()
        for net in (a, b):
            net.train_step(x, t, 30, 1e-3, mode=1, scale=0.7)
        for name in ('dw', 'db', 'w', 'b', 'wb', 'wt', 'm', 'v', 'bb', 'mb', 'vb'):
            for u, v in zip(getattr(a, name), getattr(b, name)):
                assert torch.equal(u, v), (m, name)
