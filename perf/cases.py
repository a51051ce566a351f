"""Performance cases: the work a training program has this framework do, each through a public entry point.

A case is a dict of plain values.  ``kind`` names the entry point:

``linear``      one FP8 linear layer (``msamp.initialize`` on an ``nn.Linear``), forward and backward
``mlp``         the MLP half of a transformer block, forward and backward (``fused_layers.mlp_sublayer``)
``attention``   softmax attention on a packed QKV projection, forward and backward (``ops.nn.attention_qkv``)
``layernorm``   LayerNorm forward and backward (``ops.nn.layer_norm``)
``head``        final LayerNorm, vocabulary projection and cross-entropy, forward and backward
``adam``        one low-bit AdamW step over the parameters of a transformer block (``optim.LBAdamW``)
``quantize``    ``tensor.fused_cast_transpose`` or ``tensor.cast`` and back
``accumulate``  gradient accumulation into an FP8 main gradient (``Arithmetic.add_to_fp8``)
``gpt``         logits of a whole GPT model without gradients

``prepare`` builds what a program holds before the call, ``run`` is one pass, ``exact`` the same pass in 64-bit torch
with the same quantisation points and none of the framework's code.
"""
import math

import torch
import torch.nn as nn

import msamp
from msamp.common.dtype import Dtypes
from msamp.common.tensor import ScalingTensor
from msamp.models import GPT
from msamp.models.gpt import GPTConfig, LayerNorm
from msamp.nn import ScalingParameter
from msamp.nn import fused_layers as FL
from msamp.operators.arithmetic import Arithmetic
from msamp.ops import nn as K
from msamp.optim import LBAdamW

DEV = 'cuda'
DTYPES = {'bf16': torch.bfloat16, 'fp16': torch.float16, 'fp32': torch.float32}
SIZE = {'bf16': 2, 'fp16': 2, 'fp32': 4}
QTYPES = {'e4m3': Dtypes.kfloat8_e4m3, 'e5m2': Dtypes.kfloat8_e5m2}
FLOAT8 = {'e4m3': torch.float8_e4m3fn, 'e5m2': torch.float8_e5m2}
QMAX = {'e4m3': 448.0, 'e5m2': 57344.0, 'fp16': 65504.0}


def listed():
    return [
        # the smallest call: fc1 of the test-size GPT on one short sequence, first steps of training (in-time scaling)
        dict(name='linear_tiny', kind='linear', tokens=128, cin=128, cout=512, dtype='bf16', bias=True, delayed=False),
        # an image batch through fc1 of ViT-B/16: 8 images of 197 tokens, ragged rows, past the warm-up (delayed scaling)
        dict(name='linear_vit', kind='linear', tokens=1576, cin=768, cout=3072, dtype='bf16', bias=True, delayed=True),
        # the MLP of one GPT-7B layer at the training benchmark's tokens per micro-batch: the largest GEMM work
        dict(name='mlp_7b', kind='mlp', tokens=8192, hidden=4096, ffn=16384, dtype='bf16', delayed=True),
        # ViT-B/16 attention: bidirectional, head size 64, 197 tokens
        dict(name='attn_vit', kind='attention', batch=64, seq=197, heads=12, dim=64, causal=False),
        # GPT-small attention: causal, head size 64
        dict(name='attn_gpt_small', kind='attention', batch=8, seq=1024, heads=12, dim=64, causal=True),
        # GPT-7B attention: causal, head size 128
        dict(name='attn_gpt_7b', kind='attention', batch=4, seq=2048, heads=32, dim=128, causal=True),
        # LayerNorm of a GPT-7B layer run as a module of its own, fp32 parameters
        dict(name='layernorm_7b', kind='layernorm', rows=8192, cols=4096, dtype='bf16', pdtype='fp32'),
        # loss of GPT-1.3B: final LayerNorm, 50304-way projection, cross-entropy
        dict(name='head_1p3b', kind='head', tokens=4096, hidden=2048, vocab=50304, dtype='bf16'),
        # optimizer step over one transformer block of hidden size 2048 (O2 states: e4m3 / scaled fp16)
        dict(name='adam_block', kind='adam', hidden=2048, opt='O2'),
        # operand of a tensor-parallel linear: e5m2 output gradient, row-major and transposed
        dict(name='quantize_transpose', kind='quantize', rows=4096, cols=5120, dtype='bf16', qtype='e5m2', transpose=True),
        # weight gradient of a tensor-parallel shard added to its FP8 main gradient
        dict(name='accumulate', kind='accumulate', rows=5120, cols=2560, dtype='fp32', qtype='e4m3'),
        # scoring one sequence with GPT-small after training (delayed scales).  Four of its layers: FP8 rounding decisions that
        # differ in the last bit of a bf16 input travel on, and more layers would leave nothing to compare
        dict(name='gpt_small_logits', kind='gpt', layers=4, heads=12, dim=64, vocab=50304, batch=1, seq=1024),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['linear', 'linear', 'mlp', 'attention', 'attention', 'layernorm', 'head', 'adam', 'quantize', 'accumulate', 'gpt'])
    if kind == 'linear':
        # rows are whatever the batch gives; features are multiples of 16 as in every model, or a classifier's 10 / 1000
        cin = 16 * _log_int(rng, 8, 576)
        cout = rng.choice([10, 1000]) if rng.random() < 0.15 else 16 * _log_int(rng, 8, 1024)
        return dict(kind=kind, tokens=_log_int(rng, 32, 16384), cin=cin, cout=cout, dtype=rng.choice(['bf16', 'bf16', 'bf16', 'fp16', 'fp32']),
                    bias=rng.random() < 0.8, delayed=rng.random() < 0.6)
    if kind == 'mlp':
        hidden = 64 * _log_int(rng, 2, 64)
        return dict(kind=kind, tokens=8 * _log_int(rng, 16, 1024), hidden=hidden, ffn=4 * hidden, dtype='bf16', delayed=rng.random() < 0.7)
    if kind == 'attention':
        seq = _log_int(rng, 33, 4096)
        heads, dim = rng.randint(2, 32), rng.choice([64, 128])
        batch = max(1, min(64, _log_int(rng, 1, max(2, 131072 // seq)), 262144 // (seq * heads)))
        return dict(kind=kind, batch=batch, seq=seq, heads=heads, dim=dim, causal=rng.random() < 0.6)
    if kind == 'layernorm':
        cols = 8 * _log_int(rng, 16, 1024)
        return dict(kind=kind, rows=_log_int(rng, 32, max(64, (1 << 26) // cols)), cols=cols, dtype=rng.choice(['bf16', 'bf16', 'fp16', 'fp32']) if cols <= 4096 else 'bf16',
                    pdtype='fp32')
    if kind == 'head':
        return dict(kind=kind, tokens=_log_int(rng, 64, 4096), hidden=64 * _log_int(rng, 2, 32), vocab=rng.choice([512, 32000, 50257 + 47, 50304]), dtype='bf16')
    if kind == 'adam':
        return dict(kind=kind, hidden=16 * _log_int(rng, 8, 192), opt=rng.choice(['O1', 'O2', 'O2']))
    if kind == 'quantize':
        return dict(kind=kind, rows=_log_int(rng, 16, 8192), cols=rng.choice([1, 8, 16]) * _log_int(rng, 16, 512), dtype=rng.choice(['bf16', 'bf16', 'fp16', 'fp32']),
                    qtype=rng.choice(['e4m3', 'e5m2']), transpose=rng.random() < 0.5)
    if kind == 'accumulate':
        return dict(kind=kind, rows=_log_int(rng, 16, 8192), cols=_log_int(rng, 16, 4096), dtype=rng.choice(['fp32', 'fp32', 'bf16']), qtype=rng.choice(['e4m3', 'e5m2']))
    seq = 8 * _log_int(rng, 4, 128)
    return dict(kind=kind, layers=rng.randint(1, 4), heads=rng.randint(2, 16), dim=rng.choice([64, 128]), vocab=rng.choice([512, 50304]), batch=rng.randint(1, max(1, 2048 // seq)),
                seq=seq)


# ------------------------------------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(1000003 * (seed % 1000003) + 17)


def _randn(g, *shape, std=1.0, dtype=torch.float32):
    return (torch.randn(*shape, generator=g, device=DEV) * std).to(dtype)


def _activations(g, rows, cols, dtype):
    """Hidden states: unit scale with per-channel gains and a few strong channels, as a trained network has them."""
    gain = torch.exp(0.3 * torch.randn(cols, generator=g, device=DEV))
    gain[::97] *= 4.0
    return (torch.randn(rows, cols, generator=g, device=DEV) * gain).to(dtype)


def _inputs(case, seed):
    """The random tensors of a case, the same for ``prepare`` and ``exact``."""
    g = _gen(seed)
    k = case['kind']
    dt = DTYPES[case.get('dtype', 'bf16')]
    if k == 'linear':
        t, ci, co = case['tokens'], case['cin'], case['cout']
        d = dict(x=_activations(g, t, ci, dt), w=_randn(g, co, ci, std=0.02), dy=_randn(g, t, co, std=1e-3, dtype=dt))
        d['b'] = _randn(g, co, std=0.1) if case['bias'] else None
        return d
    if k == 'mlp':
        t, h, f = case['tokens'], case['hidden'], case['ffn']
        return dict(x=_activations(g, t, h, dt), lw=1 + _randn(g, h, std=0.1), lb=_randn(g, h, std=0.05), w1=_randn(g, f, h, std=0.02), b1=_randn(g, f, std=0.05),
                    w2=_randn(g, h, f, std=0.01), b2=_randn(g, h, std=0.05), dy=_randn(g, t, h, std=1e-3, dtype=dt))
    if k == 'attention':
        shape = (case['batch'], case['seq'], 3, case['heads'], case['dim'])
        qkv = _randn(g, *shape, dtype=dt)
        return dict(qkv=qkv, do=_randn(g, case['batch'], case['seq'], case['heads'], case['dim'], std=1e-2, dtype=dt))
    if k == 'layernorm':
        r, c = case['rows'], case['cols']
        return dict(x=_activations(g, r, c, dt), w=1 + _randn(g, c, std=0.1), b=_randn(g, c, std=0.05), dy=_randn(g, r, c, std=1e-2, dtype=dt))
    if k == 'head':
        t, h, v = case['tokens'], case['hidden'], case['vocab']
        return dict(x=_activations(g, t, h, dt), lw=1 + _randn(g, h, std=0.1), lb=_randn(g, h, std=0.05), w=_randn(g, v, h, std=0.02),
                    labels=torch.randint(0, v, (t, ), generator=g, device=DEV))
    if k == 'adam':
        h = case['hidden']
        names = [('qkv', (3 * h, h)), ('proj', (h, h)), ('fc1', (4 * h, h)), ('fc2', (h, 4 * h)), ('b_qkv', (3 * h, )), ('b_proj', (h, )), ('b_fc1', (4 * h, )),
                 ('b_fc2', (h, )), ('ln', (h, ))]
        return {n: dict(p=_randn(g, *s, std=0.02), g=_randn(g, *s, std=1e-4), m=_randn(g, *s, std=3e-5), v=_randn(g, *s, std=1e-4).square() + 1e-12) for n, s in names}
    if k == 'quantize':
        return dict(x=_activations(g, case['rows'], case['cols'], dt))
    if k == 'accumulate':
        r, c = case['rows'], case['cols']
        return dict(main=_randn(g, r, c, std=1e-3), grad=_randn(g, r, c, std=1e-3, dtype=dt))
    h, v = case['heads'] * case['dim'], case['vocab']
    # as in a trained network, the residual stream is large beside what one block adds to it
    d = {'wte.weight': _randn(g, v, h, std=2.0, dtype=dt), 'wpe.weight': _randn(g, case['seq'], h, std=1.0, dtype=dt)}
    small = 0.02 / math.sqrt(2 * case['layers'])
    for i in range(case['layers']):
        for ln in ('ln1', 'ln2'):
            d[f'blocks.{i}.{ln}.weight'] = 1 + _randn(g, h, std=0.1)
            d[f'blocks.{i}.{ln}.bias'] = _randn(g, h, std=0.05)
        for n, (o, c) in dict(qkv=(3 * h, h), proj=(h, h), fc1=(4 * h, h), fc2=(h, 4 * h)).items():
            d[f'blocks.{i}.{n}.weight'] = _randn(g, o, c, std=small if n in ('proj', 'fc2') else 0.02)
            d[f'blocks.{i}.{n}.bias'] = _randn(g, o, std=0.02)
    d['ln_f.weight'], d['ln_f.bias'] = 1 + _randn(g, h, std=0.1), _randn(g, h, std=0.05)
    d['lm_head.weight'] = _randn(g, v, h, std=0.02)
    return d, torch.randint(0, v, (case['batch'], case['seq']), generator=g, device=DEV)


class _Mlp(nn.Module):
    def __init__(self, h, f):
        super().__init__()
        self.ln = LayerNorm(h, device=DEV)
        self.fc1, self.fc2 = nn.Linear(h, f, device=DEV), nn.Linear(f, h, device=DEV)

    def forward(self, x):
        return FL.mlp_sublayer(x, self.ln, self.fc1, self.fc2)


class _Head(nn.Module):
    def __init__(self, h, v):
        super().__init__()
        self.ln, self.lm_head = LayerNorm(h, device=DEV), nn.Linear(h, v, bias=False, device=DEV)

    def forward(self, x, labels):
        return K.cross_entropy(FL.ln_linear(x, self.ln, self.lm_head), labels)


def _load(module, values):
    with torch.no_grad():
        for name, p in module.named_parameters():
            p.copy_(values[name])
    return msamp.initialize(module, torch.optim.AdamW(module.parameters()), opt_level='O2')[0]


def _warm(model):
    """End the warm-up of every layer: from here on the scales of the recorded history are used (delayed scaling)."""
    for m in model.modules():
        for meta in getattr(m, 'scaling_metas', {}).values():
            meta.amax_counter.fill_(meta.window_size)


def prepare(case, seed):
    k = case['kind']
    if k == 'gpt':
        values, tokens = _inputs(case, seed)
        h = case['heads'] * case['dim']
        cfg = GPTConfig(n_layer=case['layers'], n_head=case['heads'], hidden=h, ffn_hidden=4 * h, vocab_size=case['vocab'], max_seq=case['seq'])
        model = _load(GPT(cfg, device=DEV), values)
        with torch.no_grad():
            model(tokens)    # records the scales, in-time
        _warm(model)
        return dict(case=case, model=model, tokens=tokens)
    d = _inputs(case, seed)
    s = dict(case=case)
    if k == 'linear':
        m = nn.Linear(case['cin'], case['cout'], bias=case['bias'], device=DEV)
        s['model'] = _load(m, dict(weight=d['w'], bias=d['b']))
        s['x'], s['dy'] = d['x'], d['dy']
    elif k == 'mlp':
        s['model'] = _load(_Mlp(case['hidden'], case['ffn']), {'ln.weight': d['lw'], 'ln.bias': d['lb'], 'fc1.weight': d['w1'], 'fc1.bias': d['b1'],
                                                               'fc2.weight': d['w2'], 'fc2.bias': d['b2']})
        s['x'], s['dy'] = d['x'], d['dy']
    elif k == 'attention':
        s.update(d)
    elif k == 'layernorm':
        s.update(x=d['x'], dy=d['dy'], w=nn.Parameter(d['w']), b=nn.Parameter(d['b']))
    elif k == 'head':
        s['model'] = _load(_Head(case['hidden'], case['vocab']), {'ln.weight': d['lw'], 'ln.bias': d['lb'], 'lm_head.weight': d['w']})
        s['x'], s['labels'] = d['x'], d['labels']
    elif k == 'adam':
        params, o1 = [], case['opt'] == 'O1'
        for t in d.values():
            p = ScalingParameter(t['p'].cast(Dtypes.kfloat16)) if t['p'].dim() == 2 else nn.Parameter(t['p'])
            p.grad = t['g'].cast(Dtypes.kfloat8_e4m3) if t['p'].dim() == 2 else t['g']
            params.append(p)
        states = dict(exp_avg_dtype=torch.float32, exp_avg_sq_dtype=torch.float32) if o1 else {}
        opt = LBAdamW(params, lr=1e-3, **states)
        for p, t in zip(params, d.values()):    # a resumed run: moments and step count as a checkpoint holds them
            m, v = (t['m'], t['v']) if o1 else (t['m'].cast(Dtypes.kfloat8_e4m3), t['v'].cast(Dtypes.kfloat16))
            opt.state[p] = dict(step=100, exp_avg=m, exp_avg_sq=v)
        s.update(params=params, opt=opt)
    elif k == 'quantize':
        s['x'] = d['x']
    elif k == 'accumulate':
        s.update(main=d['main'].cast(QTYPES[case['qtype']]), grad=d['grad'])
    if case.get('delayed'):
        run(s)    # records the scales, in-time
        _warm(s['model'])
    return s


def _clear(model):
    for p in model.parameters():
        p.grad = None


def _weight_grad(p):
    return [p.grad.value, p.grad.meta.scale_inv]


def run(s):
    case = s['case']
    k = case['kind']
    if k == 'linear':
        m = s['model']
        _clear(m)
        x = s['x'].detach().requires_grad_(True)
        y = m(x)
        y.backward(s['dy'])
        return dict(y=y, dx=x.grad, dw=_weight_grad(m.weight), db=m.bias.grad if case['bias'] else None)
    if k == 'mlp':
        m = s['model']
        _clear(m)
        x = s['x'].detach().requires_grad_(True)
        y = m(x)
        y.backward(s['dy'])
        return dict(y=y, dx=x.grad, dlw=m.ln.weight.grad, dlb=m.ln.bias.grad, dw1=_weight_grad(m.fc1.weight), db1=m.fc1.bias.grad, dw2=_weight_grad(m.fc2.weight),
                    db2=m.fc2.bias.grad)
    if k == 'attention':
        qkv = s['qkv'].detach().requires_grad_(True)
        o = K.attention_qkv(qkv, causal=case['causal'])
        o.backward(s['do'])
        return dict(o=o, dqkv=qkv.grad)
    if k == 'layernorm':
        s['w'].grad = s['b'].grad = None
        x = s['x'].detach().requires_grad_(True)
        y = K.layer_norm(x, s['w'], s['b'])
        y.backward(s['dy'])
        return dict(y=y, dx=x.grad, dw=s['w'].grad, db=s['b'].grad)
    if k == 'head':
        m = s['model']
        _clear(m)
        x = s['x'].detach().requires_grad_(True)
        loss = m(x, s['labels'])
        loss.backward()
        return dict(loss=loss, dx=x.grad, dlw=m.ln.weight.grad, dlb=m.ln.bias.grad, dw=_weight_grad(m.lm_head.weight))
    if k == 'adam':
        s['opt'].step()
        out = []
        for p in s['params']:
            st = s['opt'].state[p]
            for t in (p, st['exp_avg'], st['exp_avg_sq']):
                out.append([t.value, t.meta.scale_inv] if isinstance(t, ScalingTensor) else t)
        return out
    if k == 'quantize':
        if case['transpose']:
            q, qt = s['x'].fused_cast_transpose(QTYPES[case['qtype']])
            return dict(q=q.value, qt=qt.value, scale_inv=q.meta.scale_inv)
        q = s['x'].cast(QTYPES[case['qtype']])
        return dict(q=q.value, scale_inv=q.meta.scale_inv, back=q.to(DTYPES[case['dtype']]))
    if k == 'accumulate':
        main = s['main']
        Arithmetic.add_to_fp8(main.value.view(-1), main.meta, s['grad'].view(-1))
        return dict(main=main.value, scale_inv=main.meta.scale_inv, amax=main.meta.amax)
    with torch.no_grad():
        return s['model'](s['tokens'])


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def work(case):
    k = case['kind']
    e = SIZE[case.get('dtype', 'bf16')]
    if k == 'linear':
        t, i, o = case['tokens'], case['cin'], case['cout']
        # x, dy in, y, dx out in the activation type; the fp16 weight's e4m3 copy in, the e4m3 gradient out
        return dict(bytes=2 * e * t * (i + o) + 2 * i * o, flops=6 * t * i * o)
    if k == 'mlp':
        t, h, f = case['tokens'], case['hidden'], case['ffn']
        return dict(bytes=4 * e * t * h + 4 * h * f, flops=12 * t * h * f)
    if k == 'attention':
        b, s, h, d = case['batch'], case['seq'], case['heads'], case['dim']
        pairs = s * (s + 1) / 2 if case['causal'] else s * s
        return dict(bytes=2 * b * s * h * d * (3 + 1 + 1 + 3), flops=14 * b * h * d * pairs)    # 2 products forward, 5 backward
    if k == 'layernorm':
        r, c = case['rows'], case['cols']
        return dict(bytes=4 * e * r * c, flops=0)
    if k == 'head':
        t, h, v = case['tokens'], case['hidden'], case['vocab']
        return dict(bytes=2 * e * t * h + 2 * h * v, flops=6 * t * h * v)
    if k == 'adam':
        n = 12 * case['hidden']**2
        return dict(bytes=n * ((2 + 1 + 2) + 5 if case['opt'] == 'O2' else (2 + 8) * 2) + n, flops=0)
    if k == 'quantize':
        n = case['rows'] * case['cols']
        return dict(bytes=n * (e + 2) if case['transpose'] else n * (2 * e + 1), flops=0)
    if k == 'accumulate':
        n = case['rows'] * case['cols']
        return dict(bytes=n * (e + 2), flops=0)
    h, t = case['heads'] * case['dim'], case['batch'] * case['seq']
    n = 12 * h * h * case['layers'] + h * case['vocab']
    return dict(bytes=n + 2 * t * case['vocab'], flops=2 * n * t + 2 * t * (case['seq'] + 1) * h * case['layers'])


def tolerance(case):
    k = case['kind']
    if k == 'quantize':
        return 'exact'
    if k == 'accumulate':
        return {'rel': 1e-6, 'differ': 1e-5}
    if k == 'adam':
        return {'rel': 1e-3, 'max': 4e-2, 'differ': 2e-3}
    if k == 'attention':
        return {'rel': 1e-2, 'max': 0.3}
    if k == 'layernorm':
        return {'rel': 4e-3 if case['dtype'] != 'fp32' else 1e-5, 'max': 0.1}
    if k == 'linear':
        return {'rel': 4e-3 if case['dtype'] != 'fp32' else 2e-4, 'max': 0.2, 'differ': 2e-3}
    if k == 'gpt':
        return {'rel': 3e-2, 'max': 0.9}
    return {'rel': 1e-2, 'max': 0.5, 'differ': 5e-3}


# ------------------------------------------------------------------------------------------------ the same passes in 64 bits
def _scale(amax, qmax):
    """Power-of-two scale of a tensor: the largest that keeps ``amax * scale`` within the format."""
    return torch.exp2(torch.floor(torch.log2(qmax / amax.double()))) if float(amax) > 0 else torch.ones((), dtype=torch.float64, device=amax.device)


def _quant(x, fmt):
    """``x`` as it is after quantisation to ``fmt`` with its own scale."""
    sc = _scale(x.abs().max(), QMAX[fmt])
    y = (x.double() * sc).clamp(-QMAX[fmt], QMAX[fmt]).float()
    return y.to(FLOAT8[fmt] if fmt in FLOAT8 else torch.float16).double() / sc


def _weight(w):
    """A weight as its e4m3 operand holds it: scaled fp16 first, then e4m3."""
    sc = _scale(w.abs().max(), QMAX['fp16'])
    w16 = (w.double() * sc).to(torch.float16).double() / sc
    s8 = _scale(w.abs().max(), QMAX['e4m3'])
    return (w16 * s8).clamp(-448, 448).float().to(torch.float8_e4m3fn).double() / s8


def _ln(x, w, b, eps=1e-5):
    x = x.double()
    mu = x.mean(1, keepdim=True)
    rstd = torch.rsqrt(x.var(1, unbiased=False, keepdim=True) + eps)
    xh = (x - mu) * rstd
    return xh * w.double() + b.double(), xh, rstd


def _ln_back(dy, xh, rstd, w):
    gd = dy * w.double()
    dx = rstd * (gd - gd.mean(1, keepdim=True) - xh * (gd * xh).mean(1, keepdim=True))
    return dx, (dy * xh).sum(0), dy.sum(0)


def _gelu(x):
    return 0.5 * x * (1 + torch.tanh(math.sqrt(2 / math.pi) * (x + 0.044715 * x**3)))


def _gelu_grad(x):
    c = math.sqrt(2 / math.pi)
    th = torch.tanh(c * (x + 0.044715 * x**3))
    return 0.5 * (1 + th) + 0.5 * x * (1 - th * th) * c * (1 + 3 * 0.044715 * x * x)


def _softmax_attention(q, k, v, causal):
    """``[heads, seq, dim]`` in 64 bits."""
    s = q @ k.transpose(1, 2) / math.sqrt(q.shape[2])
    if causal:
        n = q.shape[1]
        s = s.masked_fill(torch.ones(n, n, dtype=torch.bool, device=q.device).triu(1), float('-inf'))
    return torch.softmax(s, -1) @ v


@torch.no_grad()
def exact(case, seed):
    k = case['kind']
    dt = DTYPES[case.get('dtype', 'bf16')]
    if k == 'gpt':
        return _exact_gpt(case, seed)
    d = _inputs(case, seed)
    if k == 'linear':
        xq, wq, dyq = _quant(d['x'], 'e4m3'), _weight(d['w']), _quant(d['dy'], 'e5m2')
        y = xq @ wq.t()
        db = None
        if case['bias']:
            y, db = y + d['b'].double(), d['dy'].double().sum(0)
        return dict(y=y, dx=dyq @ wq, dw=[None, None], db=db)
    if k == 'mlp':
        y, xh, rstd = _ln(d['x'], d['lw'], d['lb'])
        yq, w1, w2 = _quant(y.to(dt), 'e4m3'), _weight(d['w1']), _weight(d['w2'])
        h = (yq @ w1.t() + d['b1'].double()).to(dt)
        gq = _quant(_gelu(h.double()).to(dt), 'e4m3')
        out = gq @ w2.t() + d['b2'].double() + d['x'].double()
        del yq, gq, y
        dyq = _quant(d['dy'], 'e5m2')
        dh = ((dyq @ w2) * _gelu_grad(h.double())).to(dt)
        dln = (_quant(dh, 'e5m2') @ w1).to(dt).double()
        dx, dlw, dlb = _ln_back(dln, xh, rstd, d['lw'])
        return dict(y=out, dx=dx + d['dy'].double(), dlw=dlw, dlb=dlb, dw1=[None, None], db1=dh.double().sum(0), dw2=[None, None], db2=d['dy'].double().sum(0))
    if k == 'attention':
        if case['batch'] * case['heads'] * case['seq']**2 * case['dim'] > 1 << 38:
            return None
        o = torch.empty(d['do'].shape, dtype=torch.float64, device=DEV)
        g = torch.empty(d['qkv'].shape, dtype=torch.float64, device=DEV)
        for b in range(case['batch']):
            leaf = d['qkv'][b].double().permute(1, 2, 0, 3).contiguous().requires_grad_(True)    # [3, heads, seq, dim]
            with torch.enable_grad():
                ob = _softmax_attention(leaf[0], leaf[1], leaf[2], case['causal'])
                gb, = torch.autograd.grad(ob, leaf, d['do'][b].double().permute(1, 0, 2))
            o[b], g[b] = ob.detach().permute(1, 0, 2), gb.permute(2, 0, 1, 3)
        return dict(o=o, dqkv=g)
    if k == 'layernorm':
        y, xh, rstd = _ln(d['x'], d['w'], d['b'])
        dx, dw, db = _ln_back(d['dy'].double(), xh, rstd, d['w'])
        return dict(y=y, dx=dx, dw=dw, db=db)
    if k == 'head':
        t = case['tokens']
        y, xh, rstd = _ln(d['x'], d['lw'], d['lb'])
        w = _weight(d['w'])
        logits = (_quant(y.to(dt), 'e4m3') @ w.t()).to(dt).double()
        lse = torch.logsumexp(logits, 1, keepdim=True)
        loss = (lse[:, 0] - logits.gather(1, d['labels'][:, None])[:, 0]).mean()
        dl = torch.exp(logits - lse)
        del logits
        dl.scatter_add_(1, d['labels'][:, None], torch.full((t, 1), -1.0, dtype=torch.float64, device=DEV))
        dl = (dl / t).to(dt)
        dln = (_quant(dl, 'e5m2') @ w).to(dt).double()
        dx, dlw, dlb = _ln_back(dln, xh, rstd, d['lw'])
        return dict(loss=loss, dx=dx, dlw=dlw, dlb=dlb, dw=[None, None])
    if k == 'adam':
        return _exact_adam(case, d)
    if k == 'quantize':
        si = 1 / _scale(d['x'].abs().max(), QMAX[case['qtype']])
        if case['transpose']:
            return dict(q=None, qt=None, scale_inv=si)
        return dict(q=None, scale_inv=si, back=_quant(d['x'], case['qtype']))
    if k == 'accumulate':
        total = _quant(d['main'], case['qtype']) + d['grad'].double()
        amax = total.abs().max()
        return dict(main=None, scale_inv=1 / _scale(amax, QMAX[case['qtype']]), amax=amax.reshape(1))
    return None


def _exact_adam(case, d):
    o1, lr, b1, b2, eps, wd, step = case['opt'] == 'O1', 1e-3, 0.9, 0.999, 1e-8, 1e-2, 101
    out = []
    for t in d.values():
        matrix = t['p'].dim() == 2
        p = _quant(t['p'], 'fp16') if matrix else t['p'].double()
        g = _quant(t['g'], 'e4m3') if matrix else t['g'].double()
        m, v = (t['m'].double(), t['v'].double()) if o1 else (_quant(t['m'], 'e4m3'), _quant(t['v'], 'fp16'))
        m = b1 * m + (1 - b1) * g
        v = b2 * v + (1 - b2) * g * g
        p = p * (1 - lr * wd) - lr / (1 - b1**step) * m / (v.sqrt() / math.sqrt(1 - b2**step) + eps)
        sp, sv = _scale(p.abs().max(), QMAX['fp16']), _scale(v.abs().max(), QMAX['fp16'])
        out.append([p * sp, 1 / sp] if matrix else p)
        out.append(m if o1 else [None, 1 / _scale(m.abs().max(), QMAX['e4m3'])])
        out.append(v if o1 else [v * sv, 1 / sv])
    return out


def _exact_gpt(case, seed):
    d, tokens = _inputs(case, seed)
    dt, b, s, nh, hd = torch.bfloat16, case['batch'], case['seq'], case['heads'], case['dim']
    h = nh * hd

    def linear(x, name):
        y = _quant(x.to(dt), 'e4m3') @ _weight(d[name + '.weight']).t()
        bias = d.get(name + '.bias')
        return y if bias is None else y + bias.double()

    x = (d['wte.weight'][tokens] + d['wpe.weight'][:s]).view(b * s, h)
    for i in range(case['layers']):
        n = f'blocks.{i}.'
        y = _ln(x, d[n + 'ln1.weight'], d[n + 'ln1.bias'])[0]
        qkv = linear(y, n + 'qkv').to(dt).double().view(b, s, 3, nh, hd).permute(0, 2, 3, 1, 4)
        o = torch.stack([_softmax_attention(q[0], q[1], q[2], True) for q in qkv])
        x = (linear(o.permute(0, 2, 1, 3).reshape(b * s, h), n + 'proj') + x.double()).to(dt)
        y = _ln(x, d[n + 'ln2.weight'], d[n + 'ln2.bias'])[0]
        a = _gelu(linear(y, n + 'fc1').to(dt).double())
        x = (linear(a, n + 'fc2') + x.double()).to(dt)
    y = _ln(x, d['ln_f.weight'], d['ln_f.bias'])[0]
    return linear(y, 'lm_head').view(b, s, -1)
