"""The work that users have this framework do, as timed cases.

Every case goes through the public Python entry points, host packing, copies
and result objects included: ``Mc.run`` on layered and voxelized media,
``Mc.sampling_volume``, ``BatchedMc.run``, ``Mlp.train_step`` and
``Surrogate.predict``.  The Monte Carlo outputs are the raw tallies, which a
seed determines bit for bit; they have no 64-bit value to be compared with.

``math`` is ``'default'`` for a simulator built without options (portable
IEEE math, the oracle's bits) and ``'native'`` for McUseNativeMath.
"""
import math
import os

import numpy as np
import torch

from pyxopto_gb300.batched import BatchedMc
from pyxopto_gb300.mcbase.mcutil import Axis
from pyxopto_gb300.mcml import mc as mcml
from pyxopto_gb300.mcml.mcutil import fiber
from pyxopto_gb300.mcvox import mc as mcvox
from pyxopto_gb300.surrogate import Mlp, Surrogate, default_weights, features, split_bf16

INF = float('inf')


def listed():
    return [
        # a quick look, or one evaluation inside an inverse-problem loop: few
        # packets, default options; the latency of one call
        {'name': 'slab_default_1e4', 'path': 'layered', 'sample': 'slab', 'math': 'default',
         'packets': 10_000, 'bins': 50, 'fluence': 0},
        # the 10 mm slab with a radial reflectance detector of the benchmark
        # configurations, at its own 1e6 packets
        {'name': 'slab_native_1e6', 'path': 'layered', 'sample': 'slab', 'math': 'native',
         'packets': 1_000_000, 'bins': 50, 'fluence': 0},
        # three-layer skin with a fluence grid under default options
        {'name': 'skin_default_2e6', 'path': 'layered', 'sample': 'skin', 'math': 'default',
         'packets': 2_000_000, 'bins': 0, 'fluence': 100},
        # the headline configuration (100^3 fluence grid) at half its packets:
        # the largest case
        {'name': 'skin_native_5e7', 'path': 'layered', 'sample': 'skin', 'math': 'native',
         'packets': 50_000_000, 'bins': 0, 'fluence': 100},
        # one point of the reference's fibre-probe sweep (its own performance
        # test): fibre source, fine radial detector, finite rmax
        {'name': 'fibre_native_1e7', 'path': 'layered', 'sample': 'fibre', 'math': 'native',
         'packets': 10_000_000, 'bins': 340, 'fluence': 0},
        # voxelized skin with a vessel on a ragged grid, default options
        {'name': 'vessel_default_1e6', 'path': 'voxels', 'math': 'default', 'packets': 1_000_000,
         'nx': 101, 'ny': 100, 'nz': 75},
        # the 200^3 skin and vessel configuration with its fluence grid
        {'name': 'vessel_native_2e7', 'path': 'voxels', 'math': 'native', 'packets': 20_000_000,
         'nx': 200, 'ny': 200, 'nz': 200},
        # photon traces, and the sampling volume of those that a detector
        # collects
        {'name': 'traces_native_5000', 'path': 'traces', 'math': 'native', 'packets': 5000,
         'maxlen': 500, 'nv': 100},
        # independent simulations over the benchmark's optical properties: a
        # small sweep and a part of a training set
        {'name': 'batched_32', 'path': 'batched', 'sims': 32, 'low': 10_000, 'high': 100_000,
         'bins': 30},
        {'name': 'batched_200', 'path': 'batched', 'sims': 200, 'low': 10_000, 'high': 1_000_000,
         'bins': 30},
        # one training step of the surrogate network at its training batch
        {'name': 'train_4096', 'path': 'train', 'batch': 4096, 'mode': 1},
        # the surrogate's inference batch
        {'name': 'predict_65536', 'path': 'predict', 'queries': 65_536},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(['layered', 'layered', 'layered', 'voxels', 'voxels', 'traces', 'batched',
                       'train', 'predict'])
    m = rng.choice(['default', 'native'])
    if path == 'layered':
        sample = rng.choice(['slab', 'skin', 'fibre'])
        top = {'slab': 5_000_000, 'skin': 20_000_000, 'fibre': 20_000_000}[sample]
        return {'path': path, 'sample': sample, 'math': m,
                'packets': _log_int(rng, 5_000, top if m == 'native' else top // 5),
                'bins': rng.randint(20, 400), 'fluence': rng.choice([0, rng.randint(20, 150)])}
    if path == 'voxels':
        return {'path': path, 'math': m,
                'packets': _log_int(rng, 20_000, 10_000_000 if m == 'native' else 2_000_000),
                'nx': _log_int(rng, 20, 200), 'ny': _log_int(rng, 20, 200), 'nz': _log_int(rng, 20, 200)}
    if path == 'traces':
        return {'path': path, 'math': m, 'packets': _log_int(rng, 500, 10_000),
                'maxlen': rng.randint(100, 500), 'nv': _log_int(rng, 20, 150)}
    if path == 'batched':
        return {'path': path, 'sims': _log_int(rng, 8, 150), 'low': 10_000,
                'high': _log_int(rng, 50_000, 1_000_000), 'bins': rng.randint(10, 100)}
    if path == 'train':
        return {'path': path, 'batch': 8 * _log_int(rng, 32, 2048), 'mode': rng.choice([0, 1])}
    return {'path': path, 'queries': _log_int(rng, 1, 200_000)}


# ------------------------------------------------------------- simulators
def _options(mod, case):
    return [mod.mcoptions.McUseNativeMath(True)] if case['math'] == 'native' else None


def _layers(mod, specs, pf, rng):
    """Layers (d, n, mua, mus, phase function arguments), with the optical
    properties of the sample varied by up to 10 %."""
    out = []
    for d, n, mua, mus, args in specs:
        s = rng.uniform(0.9, 1.1, 2)
        out.append(mod.mclayer.Layer(d=d, n=n, mua=mua * s[0], mus=mus * s[1], pf=pf(*args)))
    return mod.mclayer.Layers(out)


def _layered(case, rng):
    mod = mcml
    det = mod.mcdetector
    nb = case['bins']
    rmax = INF
    if case['sample'] == 'slab':
        layers = _layers(mod, [(0.0, 1.0, 0.0, 0.0, (0.0,)), (10e-3, 1.33, 100.0, 1e4, (0.8,)),
                               (0.0, 1.0, 0.0, 0.0, (0.0,))], mod.mcpf.Hg, rng)
        source = mod.mcsource.Line()
        dets = det.Detectors(top=det.Radial(det.Axis(0.0, 5e-3, nb)), specular=det.Total())
    elif case['sample'] == 'skin':
        layers = _layers(mod, [(0.0, 1.0, 0.0, 0.0, (0.0, 0.5)), (1e-4, 1.45, 500.0, 4e4, (0.9, 0.5)),
                               (1.5e-3, 1.40, 50.0, 2.5e4, (0.85, 0.5)), (8e-3, 1.40, 20.0, 2e4, (0.8, 0.5)),
                               (0.0, 1.0, 0.0, 0.0, (0.0, 0.5))], mod.mcpf.Gk, rng)
        source = mod.mcsource.Line()
        top = det.Radial(det.Axis(0.0, 5e-3, nb)) if nb else det.Total()
        dets = det.Detectors(top=top, bottom=det.Total(), specular=det.Total())
    else:
        layers = _layers(mod, [(INF, 1.452, 0.0, 0.0, (0.85,)), (8e-3, 1.33, 250.0, 10_000.0, (0.85,)),
                               (INF, 1.33, 0.0, 0.0, (0.85,))], mod.mcpf.Hg, rng)
        source = mod.mcsource.UniformFiberNI(fiber.MultimodeFiber(200e-6, 200e-6, 1.452, 0.22))
        dets = det.Detectors(top=det.Radial(det.RadialAxis(0.0, 1.7e-3, nb), cosmin=0.98845494))
        rmax = 5e-3
    flu = None
    if case['fluence']:
        n = case['fluence']
        A = mod.mcfluence.Axis
        flu = mod.mcfluence.Fluence(A(-5e-3, 5e-3, n), A(-5e-3, 5e-3, n), A(0.0, 10e-3, n))
    sim = mod.Mc(layers, source, dets, fluence=flu, options=_options(mod, case),
                 rnginit=int(rng.integers(1, 1 << 31)))
    sim.rmax = rmax
    return sim


def _voxels(case, rng):
    """Skin with a vessel: epidermis over a dermis-like background, a
    cylinder of blood along y, Gaussian beam, deposition on the voxel grid."""
    mod = mcvox
    A = mod.mcdetector.Axis
    half, depth = 5e-3, 10e-3
    x, y = A(-half, half, case['nx']), A(-half, half, case['ny'])
    z = A(0.0, depth, case['nz'])
    s = rng.uniform(0.9, 1.1, (3, 2))
    pf = mod.mcpf.Hg
    mats = [mod.mcmaterial.Material(n=1.0, mua=0.0, mus=0.0, pf=pf(0.0)),
            mod.mcmaterial.Material(n=1.33, mua=20.0 * s[0, 0], mus=1.5e4 * s[0, 1], pf=pf(0.9)),
            mod.mcmaterial.Material(n=1.33, mua=1657.24 * s[1, 0], mus=37593.98 * s[1, 1], pf=pf(0.9)),
            mod.mcmaterial.Material(n=1.33, mua=2000.0 * s[2, 0], mus=9398.5 * s[2, 1], pf=pf(0.9))]
    vox = mod.mcgeometry.Voxels(x, y, z)
    m = np.ones((case['nz'], case['ny'], case['nx']), np.uint8)
    m[z.centers < 1e-4] = 2
    r2 = x.centers[None, :] ** 2 + (z.centers[:, None] - 1e-3 * rng.uniform(0.9, 1.1)) ** 2
    m[np.broadcast_to((r2 <= (5e-4) ** 2)[:, None, :], m.shape)] = 3
    vox.material[...] = m
    det = mod.mcdetector
    F = mod.mcfluence
    flu = F.Fluence(F.Axis(-half, half, case['nx']), F.Axis(-half, half, case['ny']),
                    F.Axis(0.0, depth, case['nz']))
    return mod.Mc(vox, mats, mod.mcsource.GaussianBeam(3e-4, clip=5.0),
                  det.Detectors(top=det.Total(), bottom=det.Total(), specular=det.Total()),
                  fluence=flu, options=_options(mod, case), rnginit=int(rng.integers(1, 1 << 31)))


def _traces(case, rng):
    mod = mcml
    layers = _layers(mod, [(0.0, 1.45, 0.0, 0.0, (0.0,)), (1e-2, 1.33, 2e2, 250e2, (0.9,)),
                           (0.0, 1.45, 0.0, 0.0, (0.0,))], mod.mcpf.Hg, rng)
    sim = mod.Mc(layers, mod.mcsource.Line(), trace=mod.mctrace.Trace(maxlen=case['maxlen']),
                 options=_options(mod, case), rnginit=int(rng.integers(1, 1 << 31)))
    sim.rmax = 1e-2
    return sim


#: the packets that a small detector around the source collects
COLLECTED = mcml.mctrace.Filter(z=(-1e-9, 1e-9), pz=(-1.0, -0.2), r=(0.0, 5e-4, (0.0, 0.0)))


# --------------------------------------------------------------- surrogate
SIZES = (4, 256, 256, 256, 30)


def _weights(seed):
    """FP32 weights and biases of the padded network, the first layer tied
    over the high and low parts of the inputs."""
    rng = np.random.default_rng(seed)
    pads = [16, 256, 256, 256, 32]
    ws, bs = [], []
    for i in range(4):
        w = np.zeros((pads[i + 1], pads[i]), np.float32)
        lim = math.sqrt(6.0 / (SIZES[i] + SIZES[i + 1]))
        w[:SIZES[i + 1], :SIZES[i]] = rng.uniform(-lim, lim, (SIZES[i + 1], SIZES[i]))
        if i == 0:
            w[:, 4:8] = w[:, :4]
        b = np.zeros(pads[i + 1], np.float32)
        b[:SIZES[i + 1]] = rng.normal(0.0, 0.05, SIZES[i + 1])
        ws.append(w)
        bs.append(b)
    return ws, bs


def _queries(n, seed):
    """Optical properties over the surrogate's ranges."""
    rng = np.random.default_rng(seed)
    return (np.exp(rng.uniform(np.log(1.0), np.log(1000.0), n)),
            np.exp(rng.uniform(np.log(500.0), np.log(5000.0), n)),
            rng.uniform(0.6, 0.95, n), rng.uniform(1.33, 1.5, n))


def _batch(case, seed):
    """Network inputs [M, 4] and targets [M, 32] (mode 0: standardised log
    profiles; mode 1: profiles relative to the mean one)."""
    m = case['batch']
    q = _queries(m, seed)
    t = np.zeros((m, 32), np.float32)
    z = np.random.default_rng(seed + 1).normal(0.0, 1.0, (m, 30))
    t[:, :30] = z if case['mode'] == 0 else np.exp(0.8 * z)
    return q, t


SCALE = 0.8
LR = 1e-3


# ---------------------------------------------------------------- the cases
def prepare(case, seed):
    rng = np.random.default_rng(seed)
    path = case['path']
    if path == 'layered':
        return {'case': case, 'sim': _layered(case, rng)}
    if path == 'voxels':
        return {'case': case, 'sim': _voxels(case, rng)}
    if path == 'traces':
        return {'case': case, 'sim': _traces(case, rng)}
    if path == 'batched':
        sims = BatchedMc.sample_sims(case['sims'], seed=seed, packets=(case['low'], case['high']))
        return {'case': case, 'bmc': BatchedMc(sims, raxis=Axis(0.0, 3e-3, case['bins']), seed=seed + 1)}
    if path == 'train':
        q, t = _batch(case, seed)
        mlp = Mlp(sizes=SIZES, batch=case['batch'])
        mlp.load_state(*_weights(seed))
        return {'case': case, 'mlp': mlp, 'x': split_bf16(features(*q)), 't': torch.from_numpy(t).cuda()}
    return {'case': case, 'sur': Surrogate.load(default_weights()), 'q': _queries(case['queries'], seed)}


def _tallies(res):
    _, fluence, detectors = res
    out = {}
    if fluence is not None:
        out['fluence'] = fluence.raw
    if detectors is not None:
        for slot in ('top', 'bottom', 'specular'):
            raw = getattr(detectors, slot).raw
            if raw.size:
                out[slot] = raw
    return out


def run(state):
    case = state['case']
    path = case['path']
    if path in ('layered', 'voxels'):
        return _tallies(state['sim'].run(case['packets']))
    if path == 'traces':
        sim = state['sim']
        trace, _, _ = sim.run(case['packets'])
        collected, dropped = COLLECTED(trace, update=False)
        A, n = mcml.mcsv.Axis, case['nv']
        sv = mcml.mcsv.SamplingVolume(A(-1e-3, 1e-3, n), A(-1e-3, 1e-3, n), A(0.0, 2e-3, n))
        sim.sampling_volume(collected, sv)
        return {'counts': trace.n, 'dropped': dropped, 'events': np.ascontiguousarray(trace.data).view(np.float32),
                'volume': sv.data, 'weight': float(sv.weight)}
    if path == 'batched':
        return state['bmc'].run()
    if path == 'train':
        mlp = state['mlp']
        loss = mlp.train_step(state['x'], state['t'], 30, LR, mode=case['mode'], scale=SCALE)
        return {'loss': loss, 'w': mlp.w, 'b': mlp.b, 'm': mlp.m, 'v': mlp.v, 'mb': mlp.mb, 'vb': mlp.vb}
    return state['sur'].predict(*state['q'])


#: interactions per packet of the nominal samples, and the FP32 operations
#: that one interaction cannot do without (path, move, absorb, scatter and
#: the random numbers; FMA = 2)
STEPS = {'slab': 280.0, 'skin': 860.0, 'fibre': 88.0, 'voxels': 250.0, 'traces': 310.0, 'batched': 1180.0}
OPS = 91.0


def work(case):
    path = case['path']
    if path == 'layered':
        n = case['fluence'] ** 3 + case['bins'] + 2
        return {'bytes': 8 * n, 'flops': case['packets'] * STEPS[case['sample']] * OPS}
    if path == 'voxels':
        n = case['nx'] * case['ny'] * case['nz']
        return {'bytes': 9 * n, 'flops': case['packets'] * STEPS['voxels'] * OPS}
    if path == 'traces':
        events = case['packets'] * min(case['maxlen'], STEPS['traces'])
        return {'bytes': 64 * events + 8 * case['nv'] ** 3,
                'flops': case['packets'] * STEPS['traces'] * OPS}
    if path == 'batched':
        mean = (case['high'] - case['low']) / math.log(case['high'] / case['low'])
        return {'bytes': case['sims'] * (40 + 8 * case['bins']),
                'flops': case['sims'] * mean * STEPS['batched'] * OPS}
    params = 4 * 256 + 2 * 256 * 256 + 256 * 30
    if path == 'train':
        # weights, both moments and the gradient; inputs and targets once
        return {'bytes': 24 * params + case['batch'] * (16 + 4 * 30), 'flops': 6 * case['batch'] * params}
    return {'bytes': case['queries'] * (32 + 8 * 30) + 2 * params, 'flops': 2 * case['queries'] * params}


def _gelu(x):
    c = math.sqrt(2.0 / math.pi)
    t = torch.tanh(c * (x + 0.044715 * x ** 3))
    grad = 0.5 * (1 + t) + 0.5 * x * (1 - t * t) * c * (1 + 3 * 0.044715 * x * x)
    return 0.5 * x * (1 + t), grad


def _normalized(q):
    """Inputs scaled to [-1, 1] over the surrogate's ranges, in FP32."""
    lims = [(np.log(1.0), np.log(1000.0)), (np.log(500.0), np.log(5000.0)), (0.6, 0.95), (1.33, 1.5)]
    cols = [np.log(q[0]), np.log(q[1]), q[2], q[3]]
    x = np.stack([(c - lo) / (hi - lo) * 2.0 - 1.0 for c, (lo, hi) in zip(cols, lims)], 1)
    return torch.from_numpy(x.astype(np.float32)).cuda()


def _exact_train(case, seed):
    q, t = _batch(case, seed)
    m = case['batch']
    x32 = _normalized(q)
    hi = x32.to(torch.bfloat16)
    lo = (x32 - hi.float()).to(torch.bfloat16)
    x = hi.double() + lo.double()
    t = torch.from_numpy(t).cuda().double()[:, :30]
    ws, bs = _weights(seed)
    w32 = [torch.from_numpy(w).cuda() for w in ws]
    w = [a.to(torch.bfloat16).double() for a in w32]
    w[0] = w[0][:, :4]
    b = [torch.from_numpy(a).cuda().double() for a in bs]
    h, slopes = [x], []
    for i in range(4):
        pre = h[-1] @ w[i].t() + b[i]
        a, s = _gelu(pre) if i < 3 else (pre, None)
        h.append(a)
        slopes.append(s)
    y = h[-1][:, :30]
    inv = 1.0 / (m * 30)
    if case['mode'] == 0:
        d = y - t
        part, g = d * d * inv, 2.0 * d * inv
    else:
        ratio = t * torch.exp(-SCALE * y)
        part = (ratio - 1.0) ** 2 * inv
        g = -2.0 * SCALE * (torch.clamp(ratio, max=4.0) - 1.0) * inv
    rows = part.sum(1)
    pad = torch.zeros((-m) % 256, dtype=rows.dtype, device=rows.device)
    loss = torch.cat([rows, pad]).reshape(-1, 256).sum(1)
    d = torch.cat([g, torch.zeros((m, 2), dtype=g.dtype, device=g.device)], 1)
    gw, gb = [None] * 4, [None] * 4
    for i in range(3, -1, -1):
        if slopes[i] is not None:
            d = d * slopes[i]
        gw[i], gb[i] = d.t() @ h[i], d.sum(0)
        d = d @ w[i]
    gw[0] = torch.cat([gw[0], gw[0], torch.zeros((256, 8), dtype=x.dtype, device=x.device)], 1)

    def adamw(p, gr):
        mo, ve = 0.1 * gr, 0.001 * gr * gr
        return p - LR * (mo / 0.1) / (torch.sqrt(ve / 0.001) + 1e-8), mo, ve

    nw = [adamw(p.double(), gr) for p, gr in zip(w32, gw)]
    nb = [adamw(p, gr) for p, gr in zip(b, gb)]
    return {'loss': loss, 'w': [a[0] for a in nw], 'b': [a[0] for a in nb], 'm': [a[1] for a in nw],
            'v': [a[2] for a in nw], 'mb': [a[1] for a in nb], 'vb': [a[2] for a in nb]}


def _exact_predict(case, seed):
    d = np.load(os.path.join('pyxopto_gb300', 'data', 'surrogate_single_layer_radial.npz'))
    h = _normalized(_queries(case['queries'], seed)).double()
    for i in range(4):
        w = torch.from_numpy(np.asarray(d['w%d' % i], np.float64)).cuda()
        b = torch.from_numpy(np.asarray(d['b%d' % i], np.float64)).cuda()
        if i == 0:
            w = w[:, :4]
        h = h @ w.t() + b
        if i < 3:
            h = _gelu(h)[0]
    mu = torch.from_numpy(np.asarray(d['mu'], np.float64)).cuda()
    return torch.exp(mu + float(d['scale'][0]) * h[:, :30]).cpu().numpy()


def exact(case, seed):
    if case['path'] == 'train':
        return _exact_train(case, seed)
    if case['path'] == 'predict':
        return _exact_predict(case, seed)
    return None
