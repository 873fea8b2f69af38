"""Kernels that may start before the one ahead of them in the stream has ended: calls in a row, each on inputs of its own, give what the same calls
give with the device waited for after each; and sums that start from zero do so in memory that held something else."""
import types

import pytest
import torch as th

pytestmark = pytest.mark.gpu
N = 64


def _bf(*shape, std=1.0):
    return (th.randn(*shape, device='cuda') * std).bfloat16()


def _ddlerp(B, T, C, D):
    from wind_rwkv.rwkv7 import ddlerp
    ins = [_bf(B, T, C), th.rand(C, device='cuda'), th.randn(4 * D, C, device='cuda') * .02, th.randn(4, C, D, device='cuda') * .02, th.rand(4, 1, 1, C, device='cuda')]
    return lambda x: ddlerp(*x), ins, [_bf(B, T, C) for _ in range(4)]


def _attn(B, T, H):
    from wind_rwkv.rwkv7 import attn, synthetic
    d = synthetic.wkv7_inputs(B, T, H, N, seed=int(th.randint(1 << 30, (1,))), dtype=th.bfloat16, device='cuda')
    return lambda x: (attn(*x, N),), [d[n] for n in 'rwkvab'], [d['dy']]


def _mixer(B, T, C):
    from wind_rwkv.rwkv7 import TimeMixer
    model = TimeMixer(types.SimpleNamespace(n_layer=4, n_head=C // N, n_embd=C), 1).cuda()
    with th.no_grad():
        for p in model.parameters():
            p.add_(th.randn_like(p) * .02)
    params = list(model.parameters())
    return lambda x: (model(x[0]),), [_bf(B, T, C)] + params, [_bf(B, T, C)]


@pytest.mark.parametrize('make,args', [(_ddlerp, (2, 130, 128, 16)), (_ddlerp, (3, 257, 192, 32)), (_ddlerp, (1, 65, 64, 64)),
                                       (_attn, (1, 130, 3)), (_attn, (3, 1003, 2)), (_mixer, (1, 65, 256)), (_mixer, (2, 515, 128))])
def test_calls_in_a_row(make, args):
    th.manual_seed(0)
    cases = [make(*args) for _ in range(4)]
    for _, ins, _ in cases:
        for t in ins:
            t.requires_grad_()

    def run(sync):
        out = []
        for f, ins, g in cases:
            poison = th.full((1 << 24,), float('nan'), device='cuda')  # what the allocator hands out next holds NaN
            del poison
            y = f(ins)
            if sync:
                th.cuda.synchronize()
            out.append((y, th.autograd.grad(y, ins, g)))
            if sync:
                th.cuda.synchronize()
        th.cuda.synchronize()
        return out
    apart, rows = run(True), [run(False) for _ in range(3)]
    for row in rows:
        for (y0, d0), (y1, d1) in zip(apart, row):
            for a, b in zip(y0, y1):
                assert th.equal(a, b)
            for a, b in zip(d0, d1):  # weight gradients are fp32 sums by atomics, in any order (and bf16 values behind them none)
                assert th.isfinite(b).all()
                assert float((a.float() - b.float()).norm()) <= 1e-5 * float(a.float().norm()) + 1e-12


@pytest.mark.parametrize('B,H', [(1, 3), (30, 32), (38, 32)])  # a CTA per chain; the ring of several chains a CTA
def test_decode_steps_in_a_row(B, H):
    """Each step reads the state that the one before it leaves in place."""
    from wind_rwkv.rwkv7 import attn_step, synthetic
    ins = [[synthetic.wkv7_inputs(B, 1, H, N, seed=i, dtype=th.bfloat16, device='cuda')[n] for n in 'rwkvab'] for i in range(12)]

    def run(sync):
        th.manual_seed(1)
        s, ys = th.randn(B, H, N, N, device='cuda') * .1, []
        for x in ins:
            ys.append(attn_step(*x, N, s, inplace=True)[0])
            if sync:
                th.cuda.synchronize()
        th.cuda.synchronize()
        return ys + [s]
    apart = run(True)
    for _ in range(5):
        assert all(th.equal(a, b) for a, b in zip(apart, run(False)))


def _queue(kind, dtype):
    """What keeps a quarter (forward) or a twelfth (backward) of the SMs busy for milliseconds, as a call that issues it."""
    from wind_rwkv.rwkv7 import attn, synthetic
    sms = th.cuda.get_device_properties(0).multi_processor_count
    H, T = (sms // 4, 8192) if kind == 'forward' else (sms // 12, 16384)
    d = synthetic.wkv7_inputs(1, T, H, N, seed=0, dtype=dtype, device='cuda')
    ins = [d[n] for n in 'rwkvab']
    if kind == 'forward':
        def call():
            with th.no_grad():
                return [attn(*ins, N) for _ in range(12)]
        return call
    for t in ins:
        t.requires_grad_()
    y = attn(*ins, N)
    return lambda: th.autograd.grad(y, ins, d['dy'], retain_graph=True)


@pytest.mark.parametrize('kind,dtype', [('forward', th.bfloat16), ('backward', th.bfloat16), ('backward', th.float32)])
def test_waiting_kernels_leave_idle_sms_to_other_streams(kind, dtype):
    """A few chains keep some SMs busy for long, with kernels queued behind them.  These must not take the idle SMs while they wait: a short
    call on another stream, whose kernel needs whole SMs, is done long before the queue (alone it takes some 20 us; it may at most have to
    wait for one and a half of the twelve forwards)."""
    from wind_rwkv.rwkv7 import attn, synthetic
    queue = _queue(kind, dtype)
    d = synthetic.wkv7_inputs(1, 64, 64, N, seed=1, dtype=th.bfloat16, device='cuda')
    ins = [d[n] for n in 'rwkvab']
    other = th.cuda.Stream()

    def once():
        start, end, done = (th.cuda.Event(enable_timing=True) for _ in range(3))
        start.record()
        keep = [queue()]
        end.record()
        with th.cuda.stream(other), th.no_grad():
            keep.append(attn(*ins, N))
            done.record()
        th.cuda.synchronize()
        return start.elapsed_time(done), start.elapsed_time(end)
    th.cuda.synchronize()
    once()  # the allocator has its blocks, the kernels are loaded
    short, whole = min(once() for _ in range(3))
    assert short < whole / (8 if kind == 'forward' else 4), f'{short:.3f} ms of {whole:.3f}'


@pytest.mark.parametrize('D', [16, 32, 64])
def test_ddlerp_sums_start_from_zero(D):
    """The backward's outputs and its scratch hold NaN before the call.  The weight gradients are fp32 sums by atomics in any order: 1e-5 of
    their norm between two calls; dx and the scratch's dpre have no such sums."""
    from wind_rwkv.rwkv7 import _lib
    lib = _lib.lib()
    th.manual_seed(D)
    B, T, C = 2, 130, 128
    x, al, L, R, be = _bf(B, T, C), _bf(C, std=.5), _bf(4 * D, C, std=.1), _bf(4, C, D, std=.1), _bf(4, C, std=.5)
    dys = [_bf(B, T, C) for _ in range(4)]
    m, y = _bf(B, T, 4 * D), _bf(4, B, T, C)
    assert lib.wkv7_ddlerp_fwd(*[t.data_ptr() for t in (x, al, L, R, be, m, y)], B, T, C, D, _lib.stream_of(x)) == 0

    def call(fill):
        def buf(*shape, dtype=th.float32):
            return th.full(shape, fill, dtype=dtype, device='cuda')
        outs = [buf(B, T, 4 * D, dtype=th.bfloat16), buf(B, T, C, dtype=th.bfloat16), buf(C), buf(4 * D, C), buf(4, C, D), buf(4, C)]
        ws = buf(lib.wkv7_ddlerp_bwd_tc_workspace_bytes(C, D) // 4)
        args = [x, al, L, R, be, m] + dys + outs + [ws]
        assert lib.wkv7_ddlerp_bwd_tc(*[t.data_ptr() for t in args], B, T, C, D, _lib.stream_of(x)) == 0
        th.cuda.synchronize()
        assert _lib.device_status() == 0
        return outs
    zero, nan = call(0.), call(float('nan'))
    assert th.equal(zero[0], nan[0]) and th.equal(zero[1], nan[1])
    for a, b in zip(zero[2:], nan[2:]):
        assert th.isfinite(b).all() and float((a - b).norm()) <= 1e-5 * float(a.norm())


def _op(kind, seed):
    """(f, outputs' gradients): f() is a whole forward and backward on inputs of its own, without torch kernels of its own between ours."""
    from wind_rwkv.rwkv7 import attn, attn_ln, expand_loras, synthetic
    th.manual_seed(seed)
    if kind in ('ddlerp', 'mixer'):
        f, ins, g = _ddlerp(2, 130, 128, 32) if kind == 'ddlerp' else _mixer(1, 65, 256)
    elif kind == 'loras':
        B, T, C, D = 2, 100, 128, 16
        ins = ([_bf(B, T, C) for _ in range(2)] + [_bf(B, T, D) for _ in range(4)] + [th.randn(C, D, device='cuda') * .1 for _ in range(4)] +
               [th.randn(C, device='cuda') * .5 for _ in range(4)])
        f, g = lambda x: expand_loras(*x, N), [_bf(B, T, C) for _ in range(4)]
    else:
        dtype = th.float32 if kind == 'attn_f32' else th.bfloat16
        B, T, H = (1, 64, 300) if kind == 'attn_cut' else (1, 512, 3) if kind == 'split' else (2, 203, 3)
        d = synthetic.wkv7_inputs(B, T, H, N, seed=seed, dtype=dtype, device='cuda', s0_std=.1)
        ins, g = [d[n] for n in 'rwkvab'], [d['dy'], th.randn(B, H, N, N, device='cuda')]
        if kind == 'split':
            def f(x):
                with th.no_grad():
                    return attn(*x, N, s0=d['s0'], return_state=True, time_split=4)
            return lambda: list(f(ins))
        if kind == 'attn_ln':
            ins += list(synthetic.attn_ln_extras(B, T, H, N, seed=seed, dtype=dtype, device='cuda'))
        ins.append(d['s0'])
        f = lambda x: (attn_ln if kind == 'attn_ln' else attn)(*x[:-1], N, s0=x[-1], return_state=True)  # noqa: E731
    for t in ins:
        t.requires_grad_()

    def run():
        y = f(ins)
        return [t.detach() for t in y] + list(th.autograd.grad(y, ins, g))
    return run


KINDS = ['ddlerp', 'loras', 'mixer', 'attn', 'attn_cut', 'attn_ln', 'attn_f32', 'split']


def _same(want, got, kind):
    for a, b in zip(want, got):
        assert th.isfinite(b.float()).all()
        if kind in ('attn', 'attn_cut', 'attn_f32', 'split'):
            assert th.equal(a, b)
        else:  # weight gradients are fp32 sums by atomics, in any order
            assert float((a.float() - b.float()).norm()) <= 1e-5 * float(a.float().norm()) + 1e-12


@pytest.mark.parametrize('kind', KINDS)
def test_back_to_back(kind):
    """Calls on inputs that were prepared beforehand, nothing else between them: one call's first kernel may start under the last one of the
    call before, on the memory that the allocator has got back from that."""
    ops = [_op(kind, i) for i in range(4)]
    want = []
    for op in ops:
        want.append(op())
        th.cuda.synchronize()
    for _ in range(3):
        got = [op() for op in ops]
        th.cuda.synchronize()
        for a, b in zip(want, got):
            _same(a, b, kind)


@pytest.mark.parametrize('kind', KINDS)
def test_two_streams(kind):
    """Two streams at once, with calls in a row on each."""
    ops = [_op(kind, i) for i in range(2)]
    want = [op() for op in ops]
    th.cuda.synchronize()
    streams = [th.cuda.Stream() for _ in ops]
    got = [[], []]
    for _ in range(4):
        for i, (s, op) in enumerate(zip(streams, ops)):
            with th.cuda.stream(s):
                got[i].append(op())
    th.cuda.synchronize()
    for i in range(2):
        for b in got[i]:
            _same(want[i], b, kind)


@pytest.mark.parametrize('kind', KINDS)
def test_captured(kind):
    """The launches recorded in a CUDA graph, twice in a row, and the graph replayed several times on new memory contents."""
    op = _op(kind, 7)
    side = th.cuda.Stream()
    with th.cuda.stream(side):
        for _ in range(2):
            want = op()
    th.cuda.synchronize()
    want = [t.clone() for t in want]
    graph = th.cuda.CUDAGraph()
    with th.cuda.graph(graph):
        got = [op(), op()]
    for _ in range(3):
        for outs in got:
            for t in outs:
                t.fill_(float('nan'))
        graph.replay()
        graph.replay()
        th.cuda.synchronize()
        for b in got:
            _same(want, b, kind)
