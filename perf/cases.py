"""Timed cases of the GEMM family: what a decoding step, a prefill and a training step ask of the public entry points.

A case is a dict of plain values. Its `kind` names the call sequence:

  call        one dense GEMM on operands that are quantised already (FP8, FP8 x FP4, FP4 x FP4 or BF16), scales either
              packed in the layout the kernels read or FP32 per 1x128 / 128x128 as a quantiser leaves them
  step        the dense projections of a layer stack, one after the other: BF16 activations are cast to FP8 and
              multiplied with FP8 weights (`cast`), or arrive as FP8 already
  heads       the batched per-head projection 'bhr,hdr->bhd', output in BF16 or quantised to FP8
  moe         m-grouped GEMM over experts, contiguous (psum) layout
  moe_masked  m-grouped GEMM over experts with a fixed number of row slots per expert and a device-side row count
  moe_mlp     the expert MLP: m-grouped FP8 x FP4 GEMM, SwiGLU with the routing weight to FP8, m-grouped FP8 x FP4 GEMM
  dgrad       gradient of the activations: the "NN" spelling, weights read in their forward layout
  wgrad       gradient of the weights: the "TN" spelling, added to an FP32 gradient buffer
  moe_wgrad   gradient of the expert weights: K holds the experts' tokens in psum layout

Operands are N(0,1) activations and N(0,1/k) weights, block-quantised; everything comes from the seed.
"""

import math
import os
import random
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), 'deepgemm-ascend_b200'))
import deep_gemm  # noqa: E402

# (N, K) of the dense projections of the benchmark's sweep
PROJECTIONS = ((2112, 7168), (24576, 1536), (32768, 512), (7168, 16384), (4096, 7168), (7168, 2048))
ALIGN = 256         # rows (or K) on which a group of the psum layout starts


def listed():
    return [
        # One token through one projection: the smallest call there is. Latency of the call and of its launches.
        {'name': 'decode_token', 'kind': 'call', 'dtype': 'fp8', 'scales': 'packed', 'm': 1, 'n': 2112, 'k': 7168, 'bias': False},
        # A decoding step of 64 sequences through the dense projections of the sweep: 230 MB of weights, so every
        # projection reads its weights from HBM; one cast and one GEMM for each.
        {'name': 'decode_step', 'kind': 'step', 'm': 64, 'cast': True},
        # The per-head up-projection of latent attention for 128 tokens and 128 heads, quantised for the FP8 GEMM behind it.
        {'name': 'decode_heads', 'kind': 'heads', 'tokens': 128, 'heads': 128, 'r': 512, 'd': 128, 'out': 'fp8'},
        # Expert GEMM of a decoding step: 32 experts with 256 row slots, 0 to 256 rows of each in use.
        {'name': 'decode_moe', 'kind': 'moe_masked', 'experts': 32, 'slots': 256, 'n': 7168, 'k': 2048, 'layout': 1234},
        # Prefill of 4096 tokens through the dense projections of the sweep, activations in FP8 already (the headline
        # benchmark's large rows).
        {'name': 'prefill_step', 'kind': 'step', 'm': 4096, 'cast': False},
        # A prefill chunk of an odd length with the scales as an FP8 quantiser leaves them: FP32 per 1x128 and 128x128,
        # a bias added.
        {'name': 'prefill_ragged', 'kind': 'call', 'dtype': 'fp8', 'scales': 'fp32', 'm': 1531, 'n': 7168, 'k': 2048, 'bias': True},
        # FP4 x FP4, the largest row that is published for that pair.
        {'name': 'prefill_fp4', 'kind': 'call', 'dtype': 'fp4', 'scales': 'packed', 'm': 4096, 'n': 7168, 'k': 16384, 'bias': False},
        # Expert GEMM of a prefill: eight experts with 0.7 to 1.3 times 8192 rows. The largest case.
        {'name': 'prefill_moe', 'kind': 'moe', 'dtype': 'fp8', 'experts': 8, 'rows': 8192, 'n': 4096, 'k': 7168, 'layout': 1234},
        # The expert MLP on a small prefill chunk: eight experts with about 512 tokens, FP4 weights.
        {'name': 'moe_mlp', 'kind': 'moe_mlp', 'experts': 8, 'rows': 512, 'hidden': 7168, 'inter': 2048, 'layout': 1234},
        # Gradient of the activations against FP4 weights in their forward layout.
        {'name': 'backward_data', 'kind': 'dgrad', 'dtype': 'mixed', 'm': 4096, 'n': 7168, 'k': 2048},
        # Gradient of a dense projection's weights in BF16, added to the FP32 gradient.
        {'name': 'backward_weight', 'kind': 'wgrad', 'dtype': 'bf16', 'tokens': 4096, 'm': 4096, 'n': 7168},
        # Gradients of eight experts' weights in FP8 with FP32 per-32 scales, written in BF16.
        {'name': 'backward_moe_weight', 'kind': 'moe_wgrad', 'dtype': 'fp8', 'experts': 8, 'rows': 2048, 'm': 4096, 'n': 7168,
         'accumulate': False, 'layout': 1234},
    ]


def _log(rng, lo, hi, multiple=1):
    """A whole number in [lo, hi], spread over its logarithm, a multiple of `multiple`."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(multiple, min(hi // multiple * multiple, int(round(v / multiple)) * multiple))


def draw(rng):
    largest = work(next(c for c in listed() if c['name'] == 'prefill_moe'))
    while True:
        case = _draw(rng)
        cost = work(case)
        # (BF16 runs at half of the FP8 rate; nothing drawn costs more than the largest listed case)
        if cost['flops'] * (2 if case.get('dtype') == 'bf16' else 1) <= largest['flops'] and cost['bytes'] <= largest['bytes']:
            return case


def _draw(rng):
    kind = rng.choice(['call', 'call', 'call', 'step', 'heads', 'moe', 'moe_masked', 'moe_mlp', 'dgrad', 'wgrad', 'moe_wgrad'])
    n, k = _log(rng, 512, 24576, 64), _log(rng, 512, 16384, 128)
    if kind == 'call':
        dtype = rng.choice(['fp8', 'fp8', 'mixed', 'fp4', 'bf16'])
        return {'kind': kind, 'dtype': dtype, 'scales': rng.choice(['packed', 'fp32']) if dtype == 'fp8' else 'packed',
                'm': _log(rng, 1, 8192), 'n': n, 'k': k, 'bias': rng.random() < 0.3}
    if kind == 'step':
        m = _log(rng, 1, 4096)
        return {'kind': kind, 'm': m, 'cast': m <= 512 or rng.random() < 0.5}
    if kind == 'heads':
        return {'kind': kind, 'tokens': _log(rng, 8, 2048, 8), 'heads': rng.choice([16, 32, 64, 128]), 'r': rng.choice([256, 512]),
                'd': 128, 'out': rng.choice(['fp8', 'bf16'])}
    experts = rng.choice([4, 8, 16, 32])
    n, k = _log(rng, 1024, 7168, 128), _log(rng, 1024, 7168, 128)
    layout = rng.randrange(1 << 16)
    if kind == 'moe':
        return {'kind': kind, 'dtype': rng.choice(['fp8', 'mixed', 'bf16']), 'experts': experts, 'rows': _log(rng, 64, 65536 // experts),
                'n': n, 'k': k, 'layout': layout}
    if kind == 'moe_masked':
        return {'kind': kind, 'experts': experts, 'slots': rng.choice([64, 128, 256, 512]), 'n': n, 'k': k, 'layout': layout}
    if kind == 'moe_mlp':
        return {'kind': kind, 'experts': experts, 'rows': _log(rng, 32, 16384 // experts), 'hidden': k, 'inter': _log(rng, 512, 3072, 128),
                'layout': layout}
    if kind == 'dgrad':
        return {'kind': kind, 'dtype': rng.choice(['fp8', 'mixed', 'bf16']), 'm': _log(rng, 128, 8192), 'n': n, 'k': k}
    if kind == 'wgrad':
        return {'kind': kind, 'dtype': rng.choice(['fp8', 'bf16']), 'tokens': _log(rng, 512, 16384), 'm': n, 'n': k}
    return {'kind': kind, 'dtype': rng.choice(['fp8', 'bf16']), 'experts': rng.choice([4, 8, 16]), 'rows': _log(rng, 128, 2048),
            'm': n, 'n': k, 'accumulate': rng.random() < 0.5, 'layout': layout}


def _groups(case):
    """Rows of every expert, and the psum layout they make: (sizes, ends, total rows)."""
    rng = random.Random(case['layout'])
    if case['kind'] == 'moe_masked':
        return [rng.randint(0, case['slots']) for _ in range(case['experts'])], None, None
    sizes = [int(rng.uniform(0.7, 1.3) * case['rows']) for _ in range(case['experts'])]
    ends, row = [], 0
    for s in sizes:
        ends.append(row + s)
        row = (row + s + ALIGN - 1) // ALIGN * ALIGN
    return sizes, ends, row


# ------------------------------------------------------------------------------------------------------------------
# Inputs
# ------------------------------------------------------------------------------------------------------------------
class _Inputs:
    def __init__(self, seed):
        self.gen = torch.Generator(device='cuda').manual_seed(seed)

    def randn(self, *shape):
        return torch.randn(shape, device='cuda', generator=self.gen)

    @staticmethod
    def _exponents(amax, top):
        """UE8M0 bytes of the smallest power of two that is at least amax / top."""
        bits = (amax.clamp(1e-4) / top).contiguous().view(torch.int32)
        return ((bits >> 23) + ((bits & 0x7FFFFF) != 0).int()).clamp(1, 254)

    def quantised(self, rows, k, sigma, dtype='fp8', gran=(1, 32), valid=None):
        """[rows, k] of N(0, sigma^2), quantised per `gran`: (data, exponent bytes int32 [rows / gran, k / gran]).
        fp8: E4M3 [rows, k]; fp4: packed E2M1 int8 [rows, k / 2]. Rows outside `valid` are zero."""
        gm, gk = gran
        out = torch.empty((rows, k if dtype == 'fp8' else k // 2), dtype=torch.uint8, device='cuda')
        exps = torch.empty((-(-rows // gm), -(-k // gk)), dtype=torch.int32, device='cuda')
        chunk = max(gm, (1 << 26) // k // gm * gm)
        for r0 in range(0, rows, chunk):
            r1 = min(rows, r0 + chunk)
            pm, pk = -(-(r1 - r0) // gm) * gm, exps.size(1) * gk
            x = torch.zeros((pm, pk), device='cuda')
            x[:r1 - r0, :k] = self.randn(r1 - r0, k) * sigma
            if valid is not None:
                x[:r1 - r0] *= valid[r0:r1, None]
            x = x.view(pm // gm, gm, pk // gk, gk)
            e = self._exponents(x.abs().amax(dim=(1, 3)), 448.0 if dtype == 'fp8' else 6.0)
            x *= ((254 - e) << 23).view(torch.float32)[:, None, :, None]
            x = x.view(pm, pk)[:r1 - r0, :k]
            exps[r0 // gm:r0 // gm + e.size(0)] = e
            if dtype == 'fp8':
                out[r0:r1] = x.to(torch.float8_e4m3fn).view(torch.uint8)
            else:
                code = torch.bucketize(x.abs(), torch.tensor([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0], device='cuda')).to(torch.uint8)
                code |= ((x < 0) & (code != 0)).to(torch.uint8) << 3
                out[r0:r1] = code[:, 0::2] | (code[:, 1::2] << 4)
        return out.view(torch.float8_e4m3fn if dtype == 'fp8' else torch.int8), exps

    @staticmethod
    def packed(exps, mn, k, gran=(1, 32)):
        """Exponent bytes -> int16 [mn, ceil(k / 64)], MN-major, two bytes an element (the layout the kernels read)."""
        e = exps.repeat_interleave(gran[0], 0)[:mn] if gran[0] > 1 else exps
        e = e.repeat_interleave(gran[1] // 32, 1) if gran[1] > 32 else e
        e = e[:, :-(-k // 32)]
        e = torch.nn.functional.pad(e, (0, e.size(1) % 2))
        return (e[:, 0::2] | (e[:, 1::2] << 8)).to(torch.int16).t().contiguous().t()

    def operand(self, rows, k, sigma, dtype, gran=(1, 32), valid=None):
        """(data, packed scales) of a K-major operand."""
        data, exps = self.quantised(rows, k, sigma, dtype, gran, valid)
        return data, self.packed(exps, rows, k, gran)

    def experts(self, g, n, k, dtype):
        """(data [g, n, k], packed scales [g, n, k / 64]) of the experts' weights."""
        parts = [self.operand(n, k, k ** -0.5, dtype) for _ in range(g)]
        data = torch.stack([p[0].view(torch.uint8) for p in parts]).view(parts[0][0].dtype)
        return data, torch.stack([p[1].t() for p in parts]).transpose(-2, -1)

    def mn_major(self, mn, k, sigma, dtype, valid=None):
        """(data [k, mn], exponent bytes [ceil(k / 32), mn]) of an operand whose contraction runs over its rows."""
        data, exps = self.quantised(mn, k, sigma, 'fp8', (1, 32), None)
        data, exps = data.view(torch.uint8).t().contiguous(), exps.t().contiguous()
        if valid is not None:
            data *= valid[:, None].to(torch.uint8)
        return data.view(torch.float8_e4m3fn), exps

    def bf16(self, *shape, sigma=1.0):
        return (self.randn(*shape) * sigma).bfloat16()


def _valid_rows(sizes, ends, rows):
    valid = torch.zeros(rows, device='cuda')
    for s, e in zip(sizes, ends):
        valid[e - s:e] = 1
    return valid


def _transpose_fp4(w):
    """Packed E2M1 [n, k / 2] (pairs along k) -> [k, n / 2] (pairs along n)."""
    u = w.view(torch.uint8)
    codes = torch.stack((u & 15, u >> 4), dim=-1).view(u.size(0), -1).t().contiguous()
    return (codes[:, 0::2] | (codes[:, 1::2] << 4)).view(torch.int8)


def prepare(case, seed):
    x, kind, dtype = _Inputs(seed), case['kind'], case.get('dtype', 'fp8')
    s = {'case': case}
    empty = lambda *shape, dt=torch.bfloat16: torch.zeros(shape, dtype=dt, device='cuda')  # noqa: E731
    if kind == 'call':
        m, n, k = case['m'], case['n'], case['k']
        s['d'] = empty(m, n)
        s['c'] = x.bf16(1, n) if case['bias'] else None
        if dtype == 'bf16':
            s['a'], s['b'] = x.bf16(m, k), x.bf16(n, k, sigma=k ** -0.5)
        elif case['scales'] == 'fp32':
            a, ea = x.quantised(m, k, 1.0, 'fp8', (1, 128))
            b, eb = x.quantised(n, k, k ** -0.5, 'fp8', (128, 128))
            s['a'], s['b'] = (a, (ea << 23).view(torch.float32)), (b, (eb << 23).view(torch.float32))
        else:
            grans = ((1, 128), (128, 128)) if dtype == 'fp8' else ((1, 32), (1, 32))
            s['a'] = x.operand(m, k, 1.0, 'fp4' if dtype == 'fp4' else 'fp8', grans[0])
            s['b'] = x.operand(n, k, k ** -0.5, 'fp8' if dtype == 'fp8' else 'fp4', grans[1])
    elif kind == 'step':
        s['layers'] = []
        for n, k in PROJECTIONS:
            a = x.bf16(case['m'], k) if case['cast'] else x.operand(case['m'], k, 1.0, 'fp8', (1, 128))
            s['layers'].append((a, x.operand(n, k, k ** -0.5, 'fp8', (128, 128)), empty(case['m'], n)))
    elif kind == 'heads':
        t, h, r, d = case['tokens'], case['heads'], case['r'], case['d']
        a, sfa = x.experts(h, t, r, 'fp8')
        s['a'] = (a.permute(1, 0, 2).contiguous(), sfa.permute(1, 0, 2))
        s['b'] = x.experts(h, d, r, 'fp8')
        if case['out'] == 'fp8':
            s['d'] = (empty(t, h, d, dt=torch.float8_e4m3fn), torch.zeros((h * d // 64, t), dtype=torch.int16, device='cuda').t())
        else:
            s['d'] = empty(t, h, d)
    elif kind in ('moe', 'moe_mlp'):
        sizes, ends, rows = _groups(case)
        valid = _valid_rows(sizes, ends, rows)
        s['psum'] = torch.tensor(ends, dtype=torch.int32, device='cuda')
        s['spans'] = [(e - z, e) for z, e in zip(sizes, ends)]
        k = case['k'] if kind == 'moe' else case['hidden']
        if dtype == 'bf16':
            s['a'] = x.bf16(rows, k) * valid[:, None].bfloat16()
            s['b'] = x.bf16(case['experts'], case['n'], k, sigma=k ** -0.5)
        else:
            s['a'] = x.operand(rows, k, 1.0, 'fp8', (1, 32), valid)
        if kind == 'moe':
            if dtype != 'bf16':
                s['b'] = x.experts(case['experts'], case['n'], k, 'fp8' if dtype == 'fp8' else 'fp4')
            s['d'] = empty(rows, case['n'])
        else:
            inter = case['inter']
            s['w1'] = x.experts(case['experts'], 2 * inter, k, 'fp4')
            s['w2'] = x.experts(case['experts'], k, inter, 'fp4')
            s['route'] = torch.rand(rows, device='cuda', generator=x.gen) + 0.25
            s['y1'], s['y2'] = empty(rows, 2 * inter), empty(rows, k)
    elif kind == 'moe_masked':
        sizes, _, _ = _groups(case)
        g, slots, n, k = case['experts'], case['slots'], case['n'], case['k']
        valid = (torch.arange(slots, device='cuda')[None] < torch.tensor(sizes, device='cuda')[:, None]).float().view(-1)
        a, ea = x.quantised(g * slots, k, 1.0, 'fp8', (1, 32), valid)
        sfa = torch.stack([x.packed(e, slots, k).t() for e in ea.view(g, slots, -1)]).transpose(-2, -1)
        s['a'], s['b'] = (a.view(g, slots, k), sfa), x.experts(g, n, k, 'fp8')
        s['d'] = empty(g, slots, n)
        s['rows'] = torch.tensor(sizes, dtype=torch.int32, device='cuda')
        s['expected'] = max(1, sum(sizes) // g)
    elif kind == 'dgrad':
        m, n, k = case['m'], case['n'], case['k']
        s['d'] = empty(m, n)
        if dtype == 'bf16':
            s['a'], s['b'] = x.bf16(m, k), x.bf16(k, n, sigma=k ** -0.5)
        else:
            s['a'] = x.operand(m, k, 1.0, 'fp8')
            b, sfb = x.operand(n, k, k ** -0.5, 'fp8' if dtype == 'fp8' else 'fp4')
            s['b'] = (_transpose_fp4(b) if dtype == 'mixed' else b.view(torch.uint8).t().contiguous().view(torch.float8_e4m3fn), sfb.t())
    elif kind == 'wgrad':
        t, m, n = case['tokens'], case['m'], case['n']
        s['d'] = x.randn(m, n)
        if dtype == 'bf16':
            s['a'], s['b'] = x.bf16(t, m, sigma=t ** -0.5), x.bf16(t, n)
        else:
            s['a'], s['b'] = [(d, x.packed(e.t(), d.size(1), t).t()) for d, e in (x.mn_major(m, t, t ** -0.5, dtype), x.mn_major(n, t, 1.0, dtype))]
    else:
        sizes, ends, rows = _groups(case)
        valid = _valid_rows(sizes, ends, rows)
        m, n = case['m'], case['n']
        s['psum'] = torch.tensor(ends, dtype=torch.int32, device='cuda')
        s['ks'] = [(z + ALIGN - 1) // ALIGN * ALIGN for z in sizes]
        s['d'] = x.randn(case['experts'], m, n) if case['accumulate'] else empty(case['experts'], m, n)
        if dtype == 'bf16':
            s['a'], s['b'] = [x.bf16(rows, w, sigma=g) * valid[:, None].bfloat16() for w, g in ((m, rows ** -0.5), (n, 1.0))]
        else:
            s['a'], s['b'] = [(d, (e << 23).view(torch.float32)) for d, e in (x.mn_major(m, rows, rows ** -0.5, dtype, valid), x.mn_major(n, rows, 1.0, dtype, valid))]
    return s


# ------------------------------------------------------------------------------------------------------------------
# One pass
# ------------------------------------------------------------------------------------------------------------------
def run(s):
    case = s['case']
    kind, dtype = case['kind'], case.get('dtype', 'fp8')
    if kind == 'call':
        if dtype == 'bf16':
            if s['c'] is None:
                deep_gemm.bf16_gemm_nt(s['a'], s['b'], s['d'])
            else:
                deep_gemm.bf16_gemm_nt(s['a'], s['b'], s['d'], s['c'])
        elif case['scales'] == 'fp32':
            deep_gemm.fp8_gemm_nt(s['a'], s['b'], s['d'], s['c'], recipe=(1, 128, 128))
        elif dtype == 'fp8':
            deep_gemm.fp8_gemm_nt(s['a'], s['b'], s['d'], s['c'])
        else:
            deep_gemm.fp8_fp4_gemm_nt(s['a'], s['b'], s['d'], s['c'])
        return s['d']
    if kind == 'step':
        for a, w, d in s['layers']:
            deep_gemm.fp8_gemm_nt(deep_gemm.cast_to_fp8(a) if case['cast'] else a, w, d)
        return [d for _, _, d in s['layers']]
    if kind == 'heads':
        deep_gemm.fp8_einsum('bhr,hdr->bhd', s['a'], s['b'], s['d'])
        return s['d']
    if kind == 'moe':
        if dtype == 'bf16':
            deep_gemm.m_grouped_bf16_gemm_nt_contiguous(s['a'], s['b'], s['d'], s['psum'])
        else:
            deep_gemm.m_grouped_fp8_fp4_gemm_nt_contiguous(s['a'], s['b'], s['d'], s['psum'])
        return s['d']
    if kind == 'moe_masked':
        deep_gemm.m_grouped_fp8_gemm_nt_masked(s['a'], s['b'], s['d'], s['rows'], s['expected'])
        return s['d']
    if kind == 'moe_mlp':
        deep_gemm.m_grouped_fp8_fp4_gemm_nt_contiguous(s['a'], s['w1'], s['y1'], s['psum'])
        h = deep_gemm.swiglu_apply_weight_to_fp8(s['y1'], s['route'], s['psum'], expert_alignment=ALIGN)
        deep_gemm.m_grouped_fp8_fp4_gemm_nt_contiguous(h, s['w2'], s['y2'], s['psum'])
        return [s['y2'][r0:r1] for r0, r1 in s['spans']]         # (the rows between the groups hold nothing)
    if kind == 'dgrad':
        if dtype == 'bf16':
            deep_gemm.bf16_gemm_nn(s['a'], s['b'], s['d'])
        else:
            deep_gemm.fp8_fp4_gemm_nn(s['a'], s['b'], s['d'])
        return s['d']
    if kind == 'wgrad':
        (deep_gemm.bf16_gemm_tn if dtype == 'bf16' else deep_gemm.fp8_gemm_tn)(s['a'], s['b'], s['d'], s['d'])
        return s['d']
    f = deep_gemm.k_grouped_bf16_gemm_tn_contiguous if dtype == 'bf16' else deep_gemm.k_grouped_fp8_gemm_tn_contiguous
    f(s['a'], s['b'], s['d'], s['ks'], s['psum'], s['d'] if case['accumulate'] else None)
    return s['d']


def _operand_bytes(rows, k, dtype):
    return rows * k * 2 if dtype == 'bf16' else rows * (k if dtype == 'fp8' else k // 2) + rows * -(-k // 32)


def work(case):
    """Bytes with each input read once and each output written once (scales as one byte per 32 values, FP32 scales as they
    are given), multiply-adds of the rows that exist."""
    kind, dtype = case['kind'], case.get('dtype', 'fp8')
    a_type, b_type = ('fp8', 'fp4') if dtype == 'mixed' else (dtype, dtype)
    if kind == 'call':
        m, n, k = case['m'], case['n'], case['k']
        scales = case['scales'] == 'fp32'
        io = _operand_bytes(m, k, a_type) + _operand_bytes(n, k, b_type) + (n * 2 if case['bias'] else 0) + m * n * 2
        if scales:
            io += 4 * m * -(-k // 128) + 4 * -(-n // 128) * -(-k // 128) - (m + n) * -(-k // 32)
        return {'bytes': io, 'flops': 2 * m * n * k}
    if kind == 'step':
        m = case['m']
        io = sum((m * k * 2 if case['cast'] else _operand_bytes(m, k, 'fp8')) + _operand_bytes(n, k, 'fp8') + m * n * 2 for n, k in PROJECTIONS)
        return {'bytes': io, 'flops': sum(2 * m * n * k for n, k in PROJECTIONS)}
    if kind == 'heads':
        t, h, r, d = case['tokens'], case['heads'], case['r'], case['d']
        out = t * h * (d + d // 32) if case['out'] == 'fp8' else t * h * d * 2
        return {'bytes': h * (_operand_bytes(t, r, 'fp8') + _operand_bytes(d, r, 'fp8')) + out, 'flops': 2 * t * h * r * d}
    if kind in ('moe', 'moe_masked'):
        sizes = _groups(case)[0]
        rows, used, n, k = sum(sizes), sum(1 for z in sizes if z), case['n'], case['k']
        return {'bytes': _operand_bytes(rows, k, a_type) + used * _operand_bytes(n, k, b_type) + rows * n * 2, 'flops': 2 * rows * n * k}
    if kind == 'moe_mlp':
        rows, g, h, i = sum(_groups(case)[0]), case['experts'], case['hidden'], case['inter']
        return {'bytes': _operand_bytes(rows, h, 'fp8') + g * (_operand_bytes(2 * i, h, 'fp4') + _operand_bytes(h, i, 'fp4')) + rows * (4 + h * 2),
                'flops': 2 * rows * 3 * i * h}
    if kind == 'dgrad':
        m, n, k = case['m'], case['n'], case['k']
        return {'bytes': _operand_bytes(m, k, a_type) + _operand_bytes(n, k, b_type) + m * n * 2, 'flops': 2 * m * n * k}
    if kind == 'wgrad':
        t, m, n = case['tokens'], case['m'], case['n']
        return {'bytes': _operand_bytes(m, t, dtype) + _operand_bytes(n, t, dtype) + 8 * m * n, 'flops': 2 * m * n * t}
    t, g, m, n = sum(_groups(case)[0]), case['experts'], case['m'], case['n']
    io = (m + n) * (t * 2 if dtype == 'bf16' else t + 4 * -(-t // 32))
    return {'bytes': io + g * m * n * (8 if case['accumulate'] else 2), 'flops': 2 * m * n * t}


def tolerance(case):
    # About four times what the path differs from float64 sums of the same operands (with the same roundings in between).
    kind = case['kind']
    if kind == 'wgrad' or case.get('accumulate'):
        return {'rel': 1.2e-5, 'max': 6e-5}      # FP32 output: measured 3.1e-6 and 1.5e-5 (BF16 operands, 4096 terms)
    if kind == 'heads' and case['out'] == 'fp8':
        # E4M3 output of a value rounded to BF16 first: a sum next to a rounding boundary takes the neighbouring code, which
        # is up to 1/8 away (measured on 128 x 128 x 128 values: one code in 2,000,000, no scale byte)
        return {'rel': 5e-4, 'max': 0.13, 'differ': 1e-4}
    return {'rel': 6.6e-3, 'max': 1.6e-2}        # BF16 output: measured 1.66e-3 and 3.9e-3, the one rounding
