"""More rows than one launch reaches are refused before anything runs."""
import ctypes as C

import pytest

from pyxopto_gb300 import _abi

MOST = {0: 65535 * 128, 1: 65535 * 64}


@pytest.fixture
def cuda_absent():
    import torch
    if torch.cuda.is_available():
        pytest.skip('made-up pointers: only where nothing can be launched')


@pytest.fixture(params=[0, 1])
def path(lib, request):
    prev = lib.mcgb_mlp_gemm_path(request.param)
    yield request.param
    lib.mcgb_mlp_gemm_path(prev)


@pytest.mark.parametrize('over', [1, 1 << 24])
def test_predict(lib, cuda_absent, path, over):
    p = _abi.McgbMlpPredict()
    p.layers, p.m, p.bins = 1, MOST[path] + over, 30
    p.widths[0], p.widths[1] = 16, 32
    p.w[0] = p.b[0] = p.queries = p.mu = p.x = p.h[0] = p.h[1] = p.z = p.profiles = 4096
    assert lib.mcgb_mlp_predict(C.byref(p), None) == _abi.E_SIZE


def test_train_step(lib, cuda_absent):
    tab = (_abi.McgbAdamwTensor * 4)()
    for i, (r, c) in enumerate(((32, 16), (1, 32), (32, 32), (1, 32))):
        t = tab[i]
        t.rows, t.cols = r, c
        t.w = t.w_bf16 = t.wt_bf16 = t.grad = t.m = t.v = 4096
    s = _abi.McgbMlpStep()
    s.tensors, s.layers, s.nv, s.step = tab, 2, 30, 1
    for i in range(2):
        s.h[i] = s.pre[i] = s.dpre[i] = 4096
    s.x = s.target = s.loss = s.scratch = 4096
    s.m, s.scratch_size = MOST[0] + 8, 1 << 62
    assert lib.mcgb_mlp_train_step(C.byref(s), None) == _abi.E_SIZE
