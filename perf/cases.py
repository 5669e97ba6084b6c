"""The work this library does for an inference engine, as cases that can be timed.

    listed()             the cases, each a dict of plain values
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  weights, activations, output buffers and scratch, as an engine holds them, on the GPU
    run(state)           one pass through the public entry points; returns the outputs
    work(case)           bytes and operations the pass cannot do without
    tolerance(case)      how far another correct implementation of the same precision may be off

Weights are seeded N(0, 0.02) bf16 matrices put through the library's own quantiser, activations N(0, 1).
Weights are declared stable, as an engine that loads them once does.  Sizes: hidden 4096, dense MLP 12288,
expert width 1536 or 2048, 144 experts top-8 and a shared one, vocabulary 154880, linear-attention projections
of 8192 rows and low-rank ones of 64 to 128.
"""
import math

import numpy as np
import torch

import __graft_entry__

P = __graft_entry__.load_package()

SIBLINGS = '4096,4096,4096,512,64,32'


def listed():
    return [
        # One decode token through the low-rank gates of a linear-attention layer: three tiny matrices that share
        # x, then two tall ones with 128 columns, each with its own input.  The smallest calls there are.
        {'name': 'lowrank decode', 'kind': 'lowrank', 'rows': 1, 'hidden': 4096, 'rank': 128, 'extra': 64, 'wide': 8192},
        # One decode token through the six fused projections that share the layer's input, four layers deep.
        {'name': 'siblings decode', 'kind': 'siblings', 'rows': 1, 'hidden': 4096, 'outs': SIBLINGS, 'layers': 4},
        # The same for a batch of five sequences (an odd batch; scratch from the caller).
        {'name': 'siblings batch 5', 'kind': 'siblings', 'rows': 5, 'hidden': 4096, 'outs': SIBLINGS, 'layers': 4},
        # The vocabulary projection of one decode token.
        {'name': 'lm head decode', 'kind': 'head', 'rows': 1, 'hidden': 4096, 'outs': 154880},
        # The dense layers' MLP, one decode token.
        {'name': 'dense mlp decode', 'kind': 'mlp', 'rows': 1, 'hidden': 4096, 'inter': 12288},
        # A MoE layer in decode: one sequence, and a small batch.
        {'name': 'moe decode', 'kind': 'moe', 'rows': 1, 'hidden': 4096, 'inter': 1536, 'experts': 144, 'topk': 8, 'zipf': False},
        {'name': 'moe batch 4', 'kind': 'moe', 'rows': 4, 'hidden': 4096, 'inter': 1536, 'experts': 144, 'topk': 8, 'zipf': False},
        # A MoE layer on a short prompt (ragged length) and on a full prefill chunk, popular experts hit more often.
        {'name': 'moe prompt 100', 'kind': 'moe', 'rows': 100, 'hidden': 4096, 'inter': 1536, 'experts': 144, 'topk': 8, 'zipf': True},
        {'name': 'moe prefill 2048', 'kind': 'moe', 'rows': 2048, 'hidden': 4096, 'inter': 1536, 'experts': 144, 'topk': 8, 'zipf': True},
        # A projection of a prefill chunk: bf16 activations quantised per token, and with exact products.
        {'name': 'gemm prefill 512', 'kind': 'gemm', 'rows': 512, 'hidden': 4096, 'outs': 12288},
        {'name': 'gemm exact 300', 'kind': 'exact', 'rows': 300, 'hidden': 4096, 'outs': 4096},
        # Requantising one matrix of a bf16 checkpoint.
        {'name': 'quantize matrix', 'kind': 'quantize', 'outs': 12288, 'hidden': 4096},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['lowrank', 'siblings', 'siblings', 'head', 'mlp', 'moe', 'moe', 'moe', 'gemm', 'gemm', 'exact', 'quantize'])
    hidden = 256 * rng.randint(4, 16)                    # 1024 .. 4096
    if kind == 'lowrank':
        return {'kind': kind, 'rows': rng.randint(1, 4), 'hidden': hidden, 'rank': rng.choice([64, 96, 128, 192]), 'extra': rng.randint(16, 128),
                'wide': rng.randint(2048, 12288)}
    if kind == 'siblings':
        outs = ','.join(str(_log_int(rng, 24, 8192)) for _ in range(rng.randint(2, 8)))
        return {'kind': kind, 'rows': rng.choice([1, 1, 2, 3, 4, 6, 7, 8]), 'hidden': hidden, 'outs': outs, 'layers': rng.randint(2, 5)}
    if kind == 'head':
        return {'kind': kind, 'rows': rng.choice([1, 1, 2, 4]), 'hidden': 256 * rng.randint(8, 16), 'outs': _log_int(rng, 30000, 154880)}
    if kind == 'mlp':
        return {'kind': kind, 'rows': _log_int(rng, 1, 512), 'hidden': hidden, 'inter': rng.choice([256 * rng.randint(8, 16), 2048 * rng.randint(2, 6)])}
    if kind == 'moe':
        rows = rng.choice([1, rng.randint(2, 8), rng.randint(9, 15), _log_int(rng, 16, 1500), _log_int(rng, 16, 1500)])
        return {'kind': kind, 'rows': rows, 'hidden': rng.choice([2048, 3072, 4096]), 'inter': rng.choice([1024, 1536, 2048]),
                'experts': rng.choice([64, 100, 144]), 'topk': rng.choice([4, 6, 8]), 'zipf': rows >= 16}
    if kind == 'gemm':
        return {'kind': kind, 'rows': _log_int(rng, 16, 2048), 'hidden': hidden, 'outs': _log_int(rng, 1000, 12288)}
    if kind == 'exact':
        return {'kind': kind, 'rows': _log_int(rng, 16, 1024), 'hidden': hidden, 'outs': _log_int(rng, 1000, 12288)}
    return {'kind': kind, 'outs': _log_int(rng, 256, 16384), 'hidden': 16 * rng.randint(64, 512)}


# ---- inputs --------------------------------------------------------------------------------------

class _Gen:
    """Seeded device tensors."""

    def __init__(self, seed):
        self.g = torch.Generator(device='cuda').manual_seed(seed)

    def normal(self, *shape, sd=1.0):
        t = torch.randn(shape, generator=self.g, device='cuda')
        return t if sd == 1.0 else t.mul_(sd)

    def bf16(self, *shape, sd):
        return self.normal(*shape, sd=sd).to(torch.bfloat16)

    def weight(self, n, k):
        return P.quantize(self.bf16(n, k, sd=0.02))


def _zipf_bias(n, rng):
    """Ranking bias that makes expert popularity fall off like Zipf(1.1) over a random order."""
    p = 1.0 / np.arange(1, n + 1) ** 1.1
    p = p[rng.permutation(n)]
    return torch.from_numpy((0.08 * np.log(p / p.mean())).astype(np.float32)).cuda()


class _PreparedLayer:
    """A MoE layer with its tensor-core tables built, which are given back with it."""

    def __init__(self, layer):
        self.layer = layer
        self.prepared = P.moe_prepare(layer)

    def __del__(self):
        if self.prepared:
            P.moe_release(self.layer)


def prepare(case, seed):
    kind, g = case['kind'], _Gen(seed)
    P.set_option(P.OPT_STABLE_WEIGHTS, 1)
    K = case['hidden']
    if kind == 'quantize':
        w = g.bf16(case['outs'], K, sd=0.02)
        return {'kind': kind, 'w': w, 'out': P.quantize(w)}
    M = case['rows']
    if kind == 'lowrank':
        r, e, n = case['rank'], case['extra'], case['wide']
        down, up = [g.weight(r, K), g.weight(r, K), g.weight(e, K)], [g.weight(n, r), g.weight(n, r)]
        x = g.normal(M, K)
        mid = [torch.empty((M, w.N), device='cuda') for w in down]
        ys = [torch.empty((M, n), device='cuda') for _ in up]
        return {'kind': kind, 'M': M, 'down': down, 'up': up, 'x': x, 'mid': mid, 'ys': ys,
                'jobs1': P.make_jobs(down, [x] * 3, mid), 'jobs2': P.make_jobs(up, mid[:2], ys)}
    if kind == 'siblings':
        outs = [int(n) for n in case['outs'].split(',')]
        x = g.normal(M, K)
        layers = []
        for _ in range(case['layers']):
            ws = [g.weight(n, K) for n in outs]
            buf = torch.empty(M * sum(outs), device='cuda')
            ys = [t.view(M, n) for t, n in zip(buf.split([M * n for n in outs]), outs)]
            layers.append((ws, buf, ys, P.make_jobs(ws, [x] * len(ws), ys)))
        return {'kind': kind, 'M': M, 'x': x, 'layers': layers, 'ws': P.split_workspace(M, K, x.device) if M > 1 else None}
    if kind == 'head':
        return {'kind': kind, 'W': g.weight(case['outs'], K), 'x': g.normal(M, K), 'y': torch.empty((M, case['outs']), device='cuda')}
    if kind == 'mlp':
        inter = case['inter']
        gate, up, down = g.weight(inter, K), g.weight(inter, K), g.weight(K, inter)
        return {'kind': kind, 'x': g.normal(M, K), 'gate': gate, 'up': up, 'down': down, 'y': torch.empty((M, K), device='cuda'),
                'ws': P.dense_mlp_workspace(M, K, inter, 'cuda')}
    if kind == 'moe':
        E, I, topk = case['experts'], case['inter'], case['topk']
        trip = [(g.weight(I, K), g.weight(I, K), g.weight(K, I)) for _ in range(E + 1)]
        router, bias = g.bf16(E, K, sd=0.02), g.normal(E, sd=0.1)
        if case['zipf']:
            bias = bias + _zipf_bias(E, np.random.RandomState(seed % (1 << 32)))
        layer = P.MoeLayer(router, bias, trip[:E], trip[E], topk, K, I)
        layer.workspace(M)
        return {'kind': kind, 'layer': _PreparedLayer(layer), 'x': g.normal(M, K), 'y': torch.empty((M, K), device='cuda'),
                'sel': torch.empty((M, topk), dtype=torch.int32, device='cuda'), 'wts': torch.empty((M, topk), device='cuda')}
    # gemm, exact
    nbytes = (P.lib().b200_nvfp4_gemm_bf16_workspace_bytes if kind == 'gemm' else P.lib().b200_nvfp4_gemm_bf16_exact_workspace_bytes)(M, K)
    return {'kind': kind, 'W': g.weight(case['outs'], K), 'x': g.bf16(M, K, sd=1.0), 'y': torch.empty((M, case['outs']), device='cuda'),
            'ws': torch.empty(nbytes, dtype=torch.uint8, device='cuda')}


def run(s):
    kind = s['kind']
    if kind == 'lowrank':
        P.gemv_multi(s['down'], s['x'], s['M'], s['mid'], jobs=s['jobs1'])
        P.gemv_multi(s['up'], s['mid'][:2], s['M'], s['ys'], jobs=s['jobs2'])
        return s['mid'][2], s['ys']
    if kind == 'siblings':
        for ws, _, ys, jobs in s['layers']:
            P.gemv_multi(ws, s['x'], s['M'], ys, jobs=jobs, ws=s['ws'])
        return [layer[1] for layer in s['layers']]
    if kind == 'head':
        return P.gemm(s['W'], s['x'], s['y'])
    if kind == 'mlp':
        return P.dense_mlp(s['x'], s['gate'], s['up'], s['down'], 10.0, s['y'], s['ws'])
    if kind == 'moe':
        return P.moe_forward(s['layer'].layer, s['x'], s['y'], s['sel'], s['wts'])
    if kind == 'gemm':
        return P.gemm_bf16(s['W'], s['x'], s['y'], s['ws'])
    if kind == 'exact':
        return P.gemm_bf16_exact(s['W'], s['x'], s['y'], s['ws'])
    W = P.quantize(s['w'], out=s['out'])
    return W.packed, W.scale, W.gscale


# ---- what a pass costs and how exact it is -------------------------------------------------------

def _nv(n, k):
    return n * k * 9 // 16 + 4


def work(case):
    kind, K = case['kind'], case['hidden']
    if kind == 'quantize':
        n = case['outs'] * K                             # the bf16 matrix once (its maximum and its codes), the triple written
        return {'bytes': 2 * n + _nv(case['outs'], K), 'flops': 0}
    M = case['rows']
    if kind == 'lowrank':
        r, e, n = case['rank'], case['extra'], case['wide']
        return {'bytes': 2 * _nv(r, K) + _nv(e, K) + 2 * _nv(n, r) + 4 * M * (K + e + 2 * n), 'flops': 2 * M * (K * (2 * r + e) + 2 * n * r)}
    if kind == 'siblings':
        n = [int(v) for v in case['outs'].split(',')]
        return {'bytes': case['layers'] * (sum(_nv(v, K) for v in n) + 4 * M * (K + sum(n))), 'flops': case['layers'] * 2 * M * K * sum(n)}
    if kind == 'mlp':
        inter = case['inter']
        return {'bytes': 2 * _nv(inter, K) + _nv(K, inter) + 8 * M * K, 'flops': 6 * M * K * inter}
    if kind == 'moe':
        E, I, topk = case['experts'], case['inter'], case['topk']
        touched = E * (1.0 - (1.0 - topk / E) ** M) + 1  # expected number of different experts, and the shared one
        return {'bytes': touched * (2 * _nv(I, K) + _nv(K, I)) + E * (2 * K + 4) + M * (8 * K + 8 * topk),
                'flops': 6 * M * (topk + 1) * K * I + 2 * M * E * K}
    n, xb = case['outs'], 4 if kind == 'head' else 2
    return {'bytes': _nv(n, K) + M * (xb * K + 4 * n), 'flops': 2 * M * n * K}


def tolerance(case):
    kind = case['kind']
    if kind == 'quantize':
        return 'exact'
    if kind == 'lowrank':
        return {'rel': 1e-3}                             # products of 128 columns run in fp16
    if kind in ('siblings', 'head'):
        return {'rel': 5e-5}                             # activations enter with 14 fractional bits of their row's maximum
    if kind == 'exact':
        return {'rel': 2e-5}                             # exact products, fp32 sums
    if kind == 'gemm':
        return {'rel': 2e-5}                             # the FP4 codes are fixed bit for bit; fp32 sums
    # mlp, moe: below 16 rows three such products in a row; from 16 rows on the intermediate row is rounded to FP4
    # again, where the last bit of a sum decides a code now and then.  Selections: ties.
    wide = case['rows'] >= 16
    return {'rel': 3e-3 if wide else 1e-4, 'differ': 1e-3}
