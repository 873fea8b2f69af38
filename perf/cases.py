"""Representative work of this package for timing: what a training or serving program calls, at the sizes it calls it with.

Every case goes through the public entry points of `wind_rwkv.rwkv7`.  `op` names the path:

  step          attn_step: one decode step of one layer for a batch of sequences, the fp32 state updated in place
  attn          attn forward and autograd backward; with `carry` an initial state goes in and the final state's gradient too
                (truncated back-propagation through time)
  attn_ln       the same with the fused GroupNorm, bonus and gate
  prefill       attn forward under no_grad from a non-zero state, the final state returned; `split` is attn's time_split
  ddlerp        token-shift interpolation, forward and backward
  expand_loras  second stages of the LoRAs, forward and backward
  mixer         the TimeMixer layer, forward and backward
  mixer_fwd     the TimeMixer layer under no_grad (prompt processing, evaluation)
"""
import math
import os
import sys
from collections import namedtuple

import torch as th

_PKG = os.path.join(os.getcwd(), 'wind-rwkv7_b200')
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from wind_rwkv.rwkv7 import TimeMixer, attn, attn_ln, attn_step, ddlerp, expand_loras, synthetic  # noqa: E402

N = 64
DTYPES = {'bf16': th.bfloat16, 'f32': th.float32}
Config = namedtuple('Config', ['n_layer', 'n_head', 'n_embd'])


def listed():
    return [
        # generation: one sequence of a 12-head model, one token; this is called once per layer and token
        dict(name='decode_1', op='step', B=1, T=1, H=12, dtype='bf16'),
        # batched serving: 200 sequences of the 1.5B shape (32 heads), one token
        dict(name='decode_200', op='step', B=200, T=1, H=32, dtype='bf16'),
        # the headline: training at the 124M shape
        dict(name='train_124m', op='attn', B=64, T=1024, H=12, dtype='bf16', carry=False),
        # a small batch of ragged documents with the state carried between windows (truncated BPTT), 16 heads
        dict(name='train_ragged_carry', op='attn', B=3, T=1003, H=16, dtype='bf16', carry=True),
        # fp32 tensors: debugging and small models trained in full precision
        dict(name='train_f32', op='attn', B=8, T=512, H=12, dtype='f32', carry=False),
        # fused attention of the 1.5B shape, training
        dict(name='train_ln_1b5', op='attn_ln', B=16, T=4096, H=32, dtype='bf16', carry=False),
        # long-context prefill of a batch at the 2.9B shape with state carry
        dict(name='prefill_2b9', op='prefill', B=8, T=65536, H=40, dtype='bf16', split=None),
        # one long document on a 12-head model, cut in time
        dict(name='prefill_one_long', op='prefill', B=1, T=65536, H=12, dtype='bf16', split=16),
        # the two ops that feed the mixer, at its training shape
        dict(name='ddlerp_768', op='ddlerp', B=32, T=1024, C=768, D=32),
        dict(name='expand_loras_768', op='expand_loras', B=32, T=1024, C=768, D=16),
        # a whole time-mixer layer, training
        dict(name='mixer_768', op='mixer', B=32, T=1024, C=768),
        # a whole time-mixer layer over one short prompt of odd length
        dict(name='mixer_prompt', op='mixer_fwd', B=1, T=515, C=2048),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    op = rng.choice(['step', 'attn', 'attn', 'attn_ln', 'prefill', 'ddlerp', 'expand_loras', 'mixer', 'mixer_fwd'])
    if op == 'step':
        return dict(op=op, B=_log_int(rng, 1, 256), T=rng.choice([1, 1, 1, 2, 4]), H=rng.choice([8, 12, 16, 32, 40]),
                    dtype=rng.choice(['bf16', 'bf16', 'f32']))
    if op in ('attn', 'attn_ln'):
        dtype = rng.choice(['bf16', 'bf16', 'bf16', 'f32'])
        H = rng.choice([8, 12, 16, 32, 40])
        T = _log_int(rng, 33, 4096)
        # chains x time up to the largest training case (fp32: an eighth of it)
        most = 16 * 4096 * 32 // (8 if dtype == 'f32' else 1)
        B = _log_int(rng, 1, max(1, min(64, most // (T * H))))
        return dict(op=op, B=B, T=T, H=H, dtype=dtype, carry=rng.choice([False, True]))
    if op == 'prefill':
        if rng.random() < 0.3:  # few chains: the sequence cut in time
            split = rng.choice([4, 8, 16])
            return dict(op=op, B=1, T=split * 16 * _log_int(rng, 32, 256), H=rng.choice([8, 12, 16]), dtype='bf16', split=split)
        H = rng.choice([12, 16, 32, 40])
        T = _log_int(rng, 64, 32768)
        B = _log_int(rng, 1, 8)
        return dict(op=op, B=B, T=T, H=H, dtype='bf16', split=None)
    C = rng.choice([512, 768, 1024, 2048])
    T = _log_int(rng, 33, 4096)
    B = _log_int(rng, 1, max(1, min(32, 32 * 1024 * 768 * 2 // (T * C))))
    if op == 'ddlerp':
        return dict(op=op, B=B, T=T, C=C, D=rng.choice([16, 32, 32, 64]))
    if op == 'expand_loras':
        return dict(op=op, B=B, T=T, C=C, D=rng.choice([16, 16, 32, 64, 128]))
    return dict(op=op, B=B, T=T, C=C)


def prepare(case, seed):
    op, B, T = case['op'], case['B'], case['T']
    dev = th.device('cuda')
    gen = th.Generator(device=dev).manual_seed(seed + 1)

    def rn(*shape, std=1.0):
        return th.randn(*shape, generator=gen, device=dev) * std

    s = dict(op=op)
    if op in ('step', 'attn', 'attn_ln', 'prefill'):
        H, dtype = case['H'], DTYPES[case['dtype']]
        d = synthetic.wkv7_inputs(B, T, H, N, seed=seed, dtype=dtype, device=dev)
        s['ins'] = [d[n] for n in 'rwkvab']
        if op in ('step', 'prefill'):
            s['s0'] = rn(B, H, N, N, std=0.1)
            s['split'] = case.get('split')
            return s
        s['gout'] = [d['dy']]
        if op == 'attn_ln':
            s['ins'] += synthetic.attn_ln_extras(B, T, H, N, seed=seed, dtype=dtype, device=dev)
        s['s0'] = None
        if case['carry']:
            s['s0'] = rn(B, H, N, N, std=0.1).requires_grad_()
            s['gout'].append(rn(B, H, N, N))
        for t in s['ins']:
            t.requires_grad_()
        s['wrt'] = s['ins'] + ([s['s0']] if case['carry'] else [])
        return s
    C = case['C']
    if op == 'ddlerp':
        D = case['D']
        s['ins'] = [rn(B, T, C).bfloat16(), th.rand(C, generator=gen, device=dev), rn(4 * D, C, std=0.02), rn(4, C, D, std=0.02),
                    th.rand(4, 1, 1, C, generator=gen, device=dev)]
        s['gout'] = [rn(B, T, C).bfloat16() for _ in range(4)]
    elif op == 'expand_loras':
        D = case['D']
        s['ins'] = ([rn(B, T, C).bfloat16() for _ in range(2)] + [rn(B, T, D).bfloat16() for _ in range(4)] +
                    [rn(C, D, std=0.1) for _ in range(4)] + [rn(C, std=0.5) for _ in range(4)])
        s['gout'] = [rn(B, T, C).bfloat16() for _ in range(4)]
    else:
        rng_state = th.get_rng_state()
        th.manual_seed(seed)
        model = TimeMixer(Config(12, C // N, C), 3).to(dev)
        th.set_rng_state(rng_state)
        with th.no_grad():  # as after some training: nothing is exactly zero any more
            for prm in model.parameters():
                prm.add_(rn(*prm.shape, std=0.02))
        s['model'] = model
        s['ins'] = [rn(B, T, C).bfloat16()]
        if op == 'mixer_fwd':
            return s
        s['ins'] = s['ins'] + list(model.parameters())
        s['gout'] = [rn(B, T, C).bfloat16()]
    for t in s['ins']:
        t.requires_grad_()
    s['wrt'] = s['ins']
    return s


def run(s):
    op, ins = s['op'], s.get('ins')
    if op == 'step':
        return attn_step(*ins, N, s['s0'], inplace=True)
    if op == 'prefill':
        with th.no_grad():
            return attn(*ins, N, s0=s['s0'], return_state=True, time_split=s['split'])
    if op == 'mixer_fwd':
        with th.no_grad():
            return s['model'](ins[0])
    if op in ('attn', 'attn_ln'):
        f = attn if op == 'attn' else attn_ln
        outs = f(*ins, N, s0=s['s0'], return_state=True) if s['s0'] is not None else (f(*ins, N),)
    elif op == 'ddlerp':
        outs = ddlerp(*ins)
    elif op == 'expand_loras':
        outs = expand_loras(*ins, N)
    else:
        outs = (s['model'](ins[0]),)
    grads = th.autograd.grad(outs, s['wrt'], s['gout'])
    return [o.detach() for o in outs], grads


# fp32 operations per (time step, head) of the recurrence: S*w 1, S a 2, + sa b 2, + v k 2, S r 2 over the 64x64 state
_FWD_FLOPS = 9 * N * N


def work(case):
    op, B, T = case['op'], case['B'], case['T']
    if op in ('step', 'attn', 'attn_ln', 'prefill'):
        H = case['H']
        row = N * (2 if case['dtype'] == 'bf16' else 4)
        th_, state = B * T * H, B * H * N * N * 4
        if op in ('step', 'prefill'):  # six inputs, y; the state in and out
            return dict(bytes=7 * row * th_ + 2 * state, flops=_FWD_FLOPS * th_)
        rows = 14 if op == 'attn' else 16  # r w k v a b (g) dy in; y and the gradients out
        return dict(bytes=rows * row * th_ + (4 * state if case['carry'] else 0), flops=3 * _FWD_FLOPS * th_)
    C, M = case['C'], B * T
    if op == 'ddlerp':  # x, four dy in; four y, dx out; two rank-D products forward, four backward (4 streams)
        D = case['D']
        return dict(bytes=2 * 10 * C * M + 4 * 2 * (8 * D * C + 5 * C), flops=3 * 2 * (2 * 4 * D * C) * M)
    if op == 'expand_loras':  # w_in, k_in, four dy in; four outputs, dw_in, dk_in out; four rank-D inputs and their gradients
        D = case['D']
        return dict(bytes=2 * (12 * C + 8 * D) * M + 4 * 2 * (4 * D * C + 4 * C), flops=3 * 2 * (4 * D * C) * M)
    r = 32 * 4 * 2 + 64 * 2 + 16 * 2 * 4 + 128 * 2  # LoRA ranks, both stages
    params = 4 * C * C + r * C + 13 * C
    flops = (2 * (4 * C * C + r * C) + (C // N) * _FWD_FLOPS) * M
    if op == 'mixer_fwd':
        return dict(bytes=2 * 2 * C * M + 4 * params, flops=flops)
    return dict(bytes=2 * 4 * C * M + 8 * params, flops=3 * flops)


def tolerance(case):
    """fp32 tensors go through products of split operands (errors of a few 1e-6 of the RMS on long sequences), decode keeps its
    state in fp32 but stores bf16 rows; everything else is bf16 in and out with TF32 or bf16 products."""
    if case.get('dtype') == 'f32':
        return dict(rel=3e-5)
    if case['op'] in ('mixer', 'mixer_fwd'):  # a chain of bf16 tensors: each op's rounding passes through the following ones
        return dict(rel=2e-2)
    return dict(rel=1e-2)
