"""What a user of this package has it do, as cases that can be timed: decoding, prefill and training of the Gated
DeltaNet token mixer, alone and with the two steps that the layer runs either side of it.

A case names a path (`"path"`) and its sizes:

* ``decode``      ``fused_recurrent_gated_delta_rule``: one new token per sequence, or a few (a short prompt, a drafted
                  continuation), with the options that the layer turns on and a fp32 state per sequence and value head.
* ``layer_step``  one decoding step of the layer: the short convolutions of q, k and v on their caches, the recurrent
                  step, the gated RMS norm.
* ``prefill``     ``chunk_gated_delta_rule`` without gradients: prompts in, outputs and final states out.
* ``train``       ``chunk_gated_delta_rule`` forward and backward.
* ``layer_train`` the layer's token mixing, forward and backward: three short convolutions with SiLU, the chunked rule
                  with its in-kernel options, the gated RMS norm.

Sizes: ``seqs`` sequences of ``tokens`` tokens each; with ``packed`` there are ``tokens`` tokens in all, cut into
``seqs`` sequences of unequal lengths (which depend on the seed, as they do from batch to batch in use); ``heads`` query
and key heads, ``heads * group`` value heads, ``dim`` for K and V.
"""
import math
import os
import random
import sys

import torch

_PKG = os.path.join(os.getcwd(), 'flash-linear-attention_b200')
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from b200gdn import (FusedRMSNormGated, ShortConvolution, chunk_gated_delta_rule,  # noqa: E402
                     fused_recurrent_gated_delta_rule)

CONV_WIDTH = 4
DTYPES = {'bf16': torch.bfloat16, 'fp32': torch.float32}


def listed():
    return [
        # one user, one token: the latency of a chat's next token
        dict(name='decode_single', path='decode', seqs=1, tokens=1, heads=16, group=1, dim=128, dtype='bf16', pool=False),
        # a serving engine's full batch, states in a pool of slots that is updated in place
        dict(name='decode_pool_256', path='decode', seqs=256, tokens=1, heads=16, group=1, dim=128, dtype='bf16', pool=True),
        # a short prompt (the layer takes the recurrent path up to 64 tokens) for a few users
        dict(name='decode_short_prompt', path='decode', seqs=4, tokens=37, heads=16, group=1, dim=128, dtype='bf16', pool=False),
        # one decoding step of a layer with grouped value heads, an ordinary serving batch
        dict(name='layer_step_32', path='layer_step', seqs=32, heads=16, group=2, dim=128),
        # a small model's prompt, the size of the smallest configuration of the benchmark
        dict(name='prefill_small', path='prefill', seqs=1, tokens=1024, heads=4, group=1, dim=64, packed=False, options=False, carry=True),
        # prompts of many users packed into one call, grouped value heads, states carried over from an earlier part
        dict(name='prefill_packed', path='prefill', seqs=12, tokens=16384, heads=16, group=2, dim=128, packed=True, options=True, carry=True),
        # one long document
        dict(name='prefill_long', path='prefill', seqs=1, tokens=65536, heads=16, group=1, dim=128, packed=False, options=True, carry=False),
        # the headline training shape, with an initial state
        dict(name='train_4x4096', path='train', seqs=4, tokens=4096, heads=16, group=1, dim=128, packed=False, options=False, carry=True),
        # a small model's training step, head dimension 64
        dict(name='train_small_d64', path='train', seqs=8, tokens=1024, heads=8, group=1, dim=64, packed=False, options=False, carry=False),
        # documents of unequal lengths packed into one training step, grouped value heads
        dict(name='train_packed_gva', path='train', seqs=16, tokens=65536, heads=16, group=2, dim=128, packed=True, options=False, carry=True),
        # the large training shape
        dict(name='train_8x8192_h32', path='train', seqs=8, tokens=8192, heads=32, group=1, dim=128, packed=False, options=False, carry=False),
        # everything that the layer does between its projections, forward and backward
        dict(name='layer_train_4x4096', path='layer_train', seqs=4, tokens=4096, heads=16, group=1, dim=128),
    ]


def _log_int(rng, lo, hi):
    """An integer from [lo, hi], spread evenly over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    path = rng.choice(['decode', 'decode', 'layer_step', 'prefill', 'prefill', 'train', 'train', 'layer_train'])
    heads, group = rng.choice([2, 4, 8, 12, 16, 32]), rng.choice([1, 1, 2, 4])
    dim = rng.choice([64, 128, 128])
    while heads * group > 32:
        heads //= 2
    hv = heads * group
    if path == 'decode':
        several = rng.random() < 0.3
        tokens = rng.randint(2, 64) if several else 1
        seqs = _log_int(rng, 1, 16) if several else _log_int(rng, 1, max(1, 256 * 16 // hv))
        return dict(path=path, seqs=seqs, tokens=tokens, heads=heads, group=group, dim=dim,
                    dtype=rng.choice(['bf16', 'bf16', 'bf16', 'fp32']), pool=rng.random() < 0.5)
    if path == 'layer_step':
        return dict(path=path, seqs=_log_int(rng, 1, 128), heads=heads, group=group, dim=dim)
    # token rows x value heads in all: up to the largest listed case of the same path
    total = {'prefill': 65536 * 16, 'train': 65536 * 32, 'layer_train': 16384 * 16}[path] // hv
    tokens = _log_int(rng, 65, min(total, 65536))
    seqs = _log_int(rng, 1, max(1, min(16, total // tokens)))
    if path == 'layer_train':
        return dict(path=path, seqs=seqs, tokens=tokens, heads=heads, group=group, dim=dim)
    packed = rng.random() < 0.5
    if packed:   # `tokens` in all
        tokens = tokens * seqs + rng.randint(0, 63)
        tokens = min(tokens, total)
        seqs = max(2, min(16, tokens // 64))
    return dict(path=path, seqs=seqs, tokens=tokens, heads=heads, group=group, dim=dim, packed=packed,
                options=rng.random() < 0.5, carry=rng.random() < 0.5)


def _bounds(seqs, tokens, seed):
    """cu_seqlens of `seqs` sequences of unequal lengths, at least one token each, `tokens` in all."""
    rng = random.Random(seed)
    shares = [rng.uniform(1.0, 32.0) for _ in range(seqs)]      # lengths spread like 256 .. 8192
    spare, acc, cu = tokens - seqs, 0.0, [0]
    for i, s in enumerate(shares):
        acc += s
        cu.append(round(spare * acc / sum(shares)) + i + 1)
    cu[-1] = tokens
    return cu


class _Maker:
    def __init__(self, seed):
        self.dev = torch.device('cuda')
        self.gen = torch.Generator(device=self.dev).manual_seed(seed)

    def normal(self, *shape, dtype=torch.float32, unit=False, scale=1.0):
        x = torch.empty(shape, dtype=torch.float32, device=self.dev).normal_(generator=self.gen)
        if unit:
            x = torch.nn.functional.normalize(x, p=2, dim=-1)
        elif scale != 1.0:
            x.mul_(scale)
        return x.to(dtype)

    def gate_parameters(self, hv):
        """A_log and dt_bias as the layer initialises them: A in [1, 16], time steps from 0.001 to 0.1."""
        a = torch.empty(hv, device=self.dev).uniform_(1.0, 16.0, generator=self.gen).log()
        dt = torch.empty(hv, device=self.dev).uniform_(math.log(1e-3), math.log(0.1), generator=self.gen).exp()
        return a, dt + torch.log(-torch.expm1(-dt))

    def mixer_inputs(self, b, t, h, hv, d, dtype, raw):
        """q, k, v, g, beta: projections and pre-activations (`raw`, what the layer hands over), or normalised q and k,
        log decays and write strengths."""
        q, k = (self.normal(b, t, h, d, dtype=dtype, unit=not raw) for _ in range(2))
        v = self.normal(b, t, hv, d, dtype=dtype)
        g, beta = self.normal(b, t, hv), self.normal(b, t, hv)
        if raw:
            g, beta = g.to(dtype), beta.to(dtype)
        else:
            g, beta = torch.nn.functional.logsigmoid(g), torch.sigmoid(beta)
        return q, k, v, g, beta


def _layer_options(a_log, dt_bias):
    return dict(use_qk_l2norm_in_kernel=True, use_gate_in_kernel=True, A_log=a_log, dt_bias=dt_bias, use_beta_sigmoid_in_kernel=True)


def prepare(case, seed):
    m = _Maker(seed)
    path, h, d = case['path'], case['heads'], case['dim']
    hv = h * case['group']
    s = {'case': case}
    if path == 'decode':
        n, t = case['seqs'], case['tokens']
        s['qkvgb'] = m.mixer_inputs(n, t, h, hv, d, DTYPES[case['dtype']], raw=True)
        s['options'] = _layer_options(*m.gate_parameters(hv))
        if case['pool']:
            slots = n + max(1, n // 8)                      # some slots belong to users who are not in this step
            s['state'] = m.normal(slots, hv, d, d, scale=0.1)
            s['indices'] = torch.randperm(slots, device=m.dev, generator=m.gen)[:n].to(torch.int32)
        else:
            s['state'] = m.normal(n, hv, d, d, scale=0.1)
        return s
    if path in ('layer_step', 'layer_train'):
        n, t = case['seqs'], case.get('tokens', 1)
        bf16 = torch.bfloat16
        s['x'] = [m.normal(n, t, c * d, dtype=bf16) for c in (h, h, hv)]
        s['convs'] = [ShortConvolution(c * d, CONV_WIDTH, activation='silu', device=m.dev, dtype=bf16) for c in (h, h, hv)]
        s['norm'] = FusedRMSNormGated(d, eps=1e-5, device=m.dev, dtype=bf16)
        with torch.no_grad():
            for conv in s['convs']:
                conv.weight.copy_(m.normal(*conv.weight.shape, dtype=bf16, scale=0.5))
            s['norm'].weight.copy_(1.0 + m.normal(d, scale=0.1))
        s['gate'] = m.normal(n, t, hv, d, dtype=bf16)
        s['gb'] = [m.normal(n, t, hv, dtype=bf16) for _ in range(2)]
        s['params'] = m.gate_parameters(hv)
        if path == 'layer_step':
            s['caches'] = [m.normal(n, c * d, CONV_WIDTH, dtype=bf16) for c in (h, h, hv)]
            s['state'] = m.normal(n, hv, d, d, scale=0.1)
        else:
            s['do'] = m.normal(n, t, hv, d, dtype=bf16)
            s['leaves'] = [x.requires_grad_(True) for x in (*s['x'], *s['gb'], s['gate'], *s['params'])]
            s['leaves'] += [conv.weight for conv in s['convs']] + [s['norm'].weight]
        return s
    n, t = case['seqs'], case['tokens']
    b = 1 if case['packed'] else n
    s['cu'] = torch.tensor(_bounds(n, t, seed), dtype=torch.int32, device=m.dev) if case['packed'] else None
    s['qkvgb'] = m.mixer_inputs(b, t, h, hv, d, torch.bfloat16, raw=case['options'])
    params = m.gate_parameters(hv) if case['options'] else ()
    s['options'] = _layer_options(*params) if case['options'] else {}
    s['state'] = m.normal(n, hv, d, d, scale=0.1) if case['carry'] else None
    if path == 'train':
        s['leaves'] = [x.requires_grad_(True) for x in (*s['qkvgb'], *params)]
        s['grads'] = [m.normal(b, t, hv, d, dtype=torch.bfloat16)]
        if case['carry']:
            s['leaves'].append(s['state'].requires_grad_(True))
            s['grads'].append(m.normal(n, hv, d, d, scale=0.1))
    return s


def _run_layer(s, step):
    case = s['case']
    h, d = case['heads'], case['dim']
    mixed = []
    for i, (x, conv) in enumerate(zip(s['x'], s['convs'])):
        y, cache = conv(x, cache=s['caches'][i] if step else None, output_final_state=step)
        if step:
            s['caches'][i] = cache
        mixed.append(y.view(*y.shape[:2], -1, d))
    op = fused_recurrent_gated_delta_rule if step else chunk_gated_delta_rule
    o, state = op(*mixed, g=s['gb'][0], beta=s['gb'][1], initial_state=s['state'] if step else None,
                  output_final_state=step, **_layer_options(*s['params']))
    return s['norm'](o, s['gate']), state


def run(state):
    s, path = state, state['case']['path']
    if path == 'decode':
        q, k, v, g, beta = s['qkvgb']
        more = {'state_indices': s['indices']} if 'indices' in s else {}
        with torch.no_grad():
            return fused_recurrent_gated_delta_rule(q, k, v, g=g, beta=beta, initial_state=s['state'], output_final_state=True,
                                                    **s['options'], **more)
    if path == 'layer_step':
        with torch.no_grad():
            y, s['state'] = _run_layer(s, True)
        return [y, s['state'], *s['caches']]
    if path == 'layer_train':
        y, _ = _run_layer(s, False)
        return [y.detach(), *torch.autograd.grad(y, s['leaves'], s['do'])]
    if path == 'prefill':
        with torch.no_grad():
            return chunk_gated_delta_rule(*s['qkvgb'], initial_state=s['state'], output_final_state=True, cu_seqlens=s['cu'], **s['options'])
    out = chunk_gated_delta_rule(*s['qkvgb'], initial_state=s['state'], output_final_state=s['state'] is not None,
                                 cu_seqlens=s['cu'], **s['options'])
    out = [x for x in out if x is not None]
    return [x.detach() for x in out] + list(torch.autograd.grad(out, s['leaves'], s['grads']))


def work(case):
    """Bytes: the inputs of every call that is made, each read once, and its results, each written once (a backward pass
    reads the inputs of its forward pass again; nothing in between is counted).  Operations: the chunked form's dense
    64-token tiles, no recomputation; for the recurrent form its three K x V passes a token."""
    path, h, d = case['path'], case['heads'], case['dim']
    hv = h * case['group']
    n, t = case['seqs'], case.get('tokens', 1)
    rows = t if case.get('packed') else n * t
    size = 4 if case.get('dtype') == 'fp32' else 2
    qkv, val = rows * (2 * h + hv) * d * size, rows * hv * d * size
    gb = 2 * rows * hv * (4 if path in ('prefill', 'train') and not case['options'] else size)
    states = n * hv * d * d * 4
    if path in ('decode', 'layer_step'):
        out = {'bytes': qkv + gb + val + 2 * states, 'flops': 6 * rows * hv * d * d}
        if path == 'layer_step':
            conv = rows * (2 * h + hv) * d * size
            out['bytes'] += 2 * conv * (1 + CONV_WIDTH) + 3 * val      # x, y and the caches; o, gate, y
            out['flops'] += rows * (2 * h + hv) * d * 2 * CONV_WIDTH
        return out
    f_fwd = 6 * d * d + 2 * 64 * 5 * d
    f_bwd = 12 * d * d + 2 * 64 * (12 * d + 128)
    carried = states if case.get('carry') else 0
    fwd = qkv + gb + val + carried + (states if path == 'prefill' or carried else 0)
    if path == 'prefill':
        return {'bytes': fwd, 'flops': rows * hv * f_fwd}
    bwd = 2 * qkv + 2 * gb + val + 2 * carried
    out = {'bytes': fwd + bwd, 'flops': rows * hv * (f_fwd + f_bwd)}
    if path == 'layer_train':
        out['bytes'] += 5 * qkv + 8 * val                              # x, y | x, dy, dx;  o, gate, y | o, gate, dy, do, dgate
        out['flops'] += rows * (2 * h + hv) * d * 6 * CONV_WIDTH
    return out


def tolerance(case):
    if case.get('dtype') == 'fp32':
        return {'rel': 2e-5}
    if case['path'] == 'decode':
        return {'rel': 5e-3}           # fp32 arithmetic, outputs rounded to bf16
    return {'rel': 1e-2}               # bf16 operands and results
