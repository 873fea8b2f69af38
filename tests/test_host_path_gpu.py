"""The eager host path in C++ (csrc/torch_ops.cpp) against the Python form of the same entry points, which torch.compile traces and which
takes what the C++ one leaves: whole layer, ragged lengths, rows of wider tensors, frozen parameters."""
import types

import pytest
import torch as th

pytestmark = pytest.mark.gpu
N = 64


class _Nothing:
    """Stands for the extension and leaves every call to the Python form."""

    def __getattr__(self, name):
        return lambda *a: None


def _python_form(monkeypatch, f):
    from wind_rwkv.rwkv7 import _lib
    with monkeypatch.context() as m:
        m.setattr(_lib, '_ext', _Nothing())
        return f()


def _close(got, want, rel):
    assert (got is None) == (want is None)
    if want is not None:
        assert got.dtype == want.dtype and got.shape == want.shape
        d, s = (got.double() - want.double()).norm().item(), want.double().norm().item()
        assert d <= rel * s + 1e-12, (d, s)


def _grads(outs, ins, seed):
    gen = th.Generator('cuda').manual_seed(seed)
    dys = [th.randn(o.shape, generator=gen, device='cuda').to(o.dtype) for o in outs]
    return th.autograd.grad(outs, [i for i in ins if i.requires_grad], dys)


@pytest.mark.parametrize('B,T,C,frozen', [(1, 1, 64, ()), (2, 17, 128, ('Wr', 'time_aaa_w1', 'gate_w1')), (3, 80, 192, ())])
def test_mixer(B, T, C, frozen, monkeypatch):
    from wind_rwkv.rwkv7 import TimeMixer
    th.manual_seed(5)
    mixer = TimeMixer(types.SimpleNamespace(n_layer=4, n_head=C // N, n_embd=C), 1).cuda()
    for name, p in mixer.named_parameters():
        p.data += 0.05 * th.randn_like(p)
        p.requires_grad_(name not in frozen)
    x = th.randn(B, T, C, device='cuda').bfloat16().requires_grad_()
    ins = [x] + list(mixer.parameters())

    def run():
        y = mixer(x)
        return [y] + list(_grads([y], ins, 6))

    got, want = run(), _python_form(monkeypatch, run)
    for g, w in zip(got, want, strict=True):
        _close(g, w, 2e-2)
    with th.no_grad():
        assert th.equal(mixer(x), got[0])


@pytest.mark.parametrize('T', [1, 15, 16, 65])
def test_expand_loras_rows_of_wider_tensors(T, monkeypatch):
    from wind_rwkv.rwkv7 import expand_loras
    B, C, D = 3, 128, 16
    th.manual_seed(T)
    big = [th.randn(B, T, C, device='cuda').bfloat16().requires_grad_() for _ in range(2)]
    wide = th.randn(B, T, 4 * D, device='cuda').bfloat16().requires_grad_()
    par = [0.3 * th.randn(C, D, device='cuda') for _ in range(4)] + [th.randn(C, device='cuda') for _ in range(4)]
    par = [p.requires_grad_() for p in par]

    def run():
        outs = expand_loras(*big, *wide.split(D, dim=2), *par, N)
        return list(outs) + list(_grads(outs, big + [wide] + par, 7))

    got, want = run(), _python_form(monkeypatch, run)
    for g, w in zip(got[:7], want[:7]):
        assert th.equal(g, w)
    for g, w in zip(got[7:], want[7:], strict=True):  # sums over rows by atomics
        _close(g, w, 1e-5)


@pytest.mark.parametrize('dtype', [th.bfloat16, th.float32])
def test_attn_state_and_slices(dtype, monkeypatch):
    from wind_rwkv.rwkv7 import attn, synthetic
    B, T, H = 2, 19, 2
    d = synthetic.wkv7_inputs(B, T, H, N, seed=3, dtype=dtype)
    ins = [d[n].cuda().requires_grad_() for n in 'rwkvab']
    s0 = th.randn(B, H, N, N, device='cuda').requires_grad_()

    def run():
        y, sT = attn(*ins, N, s0=s0, return_state=True)
        first, = _grads([y[:, :, ::2]], ins[:1], 8),   # gradient of y alone, from a strided view
        return [y, sT] + list(first) + list(_grads(list(attn(*ins, N, s0=s0, return_state=True)), ins + [s0], 9))

    for g, w in zip(run(), _python_form(monkeypatch, run), strict=True):
        assert th.equal(g, w)


def _layouts(t, B, T, HC):
    """[B,T,HC] views of the flat tensor t: windows that overlap by half, one sequence expanded to a batch, time outside the batch."""
    return {'windows': t.as_strided((B, T, HC), (T // 2 * HC, HC, 1)), 'expanded': t.as_strided((B, T, HC), (0, HC, 1)),
            'sliding': t.as_strided((B, T, HC), (HC, HC, 1)), 'time first': t.as_strided((B, T, HC), (HC, B * HC, 1)),
            'halves': t.as_strided((B, T, HC), (T * 2 * HC, 2 * HC, 1))}


@pytest.mark.parametrize('form', ['c++', 'python'])
@pytest.mark.parametrize('layout', ['windows', 'expanded', 'sliding', 'time first', 'halves'])
def test_layouts(layout, form, monkeypatch):
    """Inputs whose rows share memory or lie in another order give what their contiguous copies give, bit for bit."""
    from wind_rwkv.rwkv7 import attn, attn_ln, attn_step, synthetic
    B, T, H = 3, 32, 2
    HC = H * N
    flat = synthetic.wkv7_inputs(1, 2 * B * T, H, N, seed=6, dtype=th.bfloat16, device='cuda')
    g, params = synthetic.attn_ln_extras(1, 2 * B * T, H, N, seed=6, dtype=th.bfloat16, device='cuda')
    s0 = th.randn(B, H, N, N, device='cuda')
    views = [_layouts(x, B, T, HC)[layout] for x in [flat[n] for n in 'rwkvab'] + [g]]

    def run(ins):
        ins = [i.detach().requires_grad_() for i in ins]
        res = [o.detach() for o in attn_step(*ins[:6], N, s0)]
        for outs in (attn(*ins[:6], N, s0=s0, return_state=True), attn_ln(*ins, params, N, s0=s0, return_state=True)):
            res += [o.detach() for o in outs] + list(_grads(list(outs), ins if len(res) > 2 else ins[:6], 11))
        return res

    want = run([v.contiguous() for v in views])
    got = run(views) if form == 'c++' else _python_form(monkeypatch, lambda: run(views))
    for a, b in zip(got, want, strict=True):
        assert th.equal(a, b)


def _ops():
    """name -> (function, inputs) of every entry point with an autograd function, at small sizes."""
    from wind_rwkv.rwkv7 import TimeMixer, attn, attn_ln, ddlerp, expand_loras, synthetic
    B, T, H, D = 2, 20, 2, 16
    C = H * N
    th.manual_seed(2)
    d = synthetic.wkv7_inputs(B, T, H, N, seed=4, dtype=th.bfloat16, device='cuda', s0_std=0.1)
    g, params = synthetic.attn_ln_extras(B, T, H, N, seed=4, dtype=th.bfloat16, device='cuda')
    x = th.randn(B, T, C, device='cuda').bfloat16()
    mixer = TimeMixer(types.SimpleNamespace(n_layer=4, n_head=H, n_embd=C), 1).cuda().requires_grad_(False)
    for p in mixer.parameters():  # (the output projection starts at zero)
        p.add_(0.05 * th.randn_like(p))
    rkv = [d[n] for n in 'rwkvab']
    par = [th.rand(C, device='cuda'), th.randn(4 * D, C, device='cuda'), th.randn(4, C, D, device='cuda'), th.rand(4, 1, 1, C, device='cuda')]
    lora = [x.flip(1)] + [th.randn(B, T, D, device='cuda').bfloat16() for _ in range(4)]
    lora += [th.randn(C, D, device='cuda') for _ in range(4)] + [th.randn(C, device='cuda') for _ in range(4)]
    return {'attn': (lambda *a: attn(*a[:6], N, s0=a[6]), rkv + [d['s0']]), 'attn_ln': (lambda *a: attn_ln(*a, N), rkv + [g, params]),
            'ddlerp': (ddlerp, [x] + par), 'expand_loras': (lambda *a: expand_loras(*a, N), [x] + lora), 'mixer': (mixer, [x])}


@pytest.mark.parametrize('op', ['attn', 'attn_ln', 'ddlerp', 'expand_loras', 'mixer'])
def test_forward_mode_raises(op):
    """No forward-mode derivative is implemented: a dual tensor in any place raises, with and without requires_grad anywhere, and
    no output comes back without its tangent."""
    import torch.autograd.forward_ad as fwd
    f, ins = _ops()[op]
    for i in {0, 1, len(ins) // 2, len(ins) - 1} & set(range(len(ins))):
        for grad in (False, True):
            with fwd.dual_level():
                dual = [fwd.make_dual(t.clone().requires_grad_(grad), th.ones_like(t)) if j == i else t for j, t in enumerate(ins)]
                with pytest.raises((NotImplementedError, RuntimeError), match='jvp'):
                    f(*dual)


@pytest.mark.parametrize('form', ['c++', 'python'])
@pytest.mark.parametrize('op', ['attn', 'attn_ln', 'ddlerp', 'expand_loras', 'mixer'])
def test_saved_tensors_come_back_in_other_layouts(op, form, monkeypatch):
    """Hooks on saved tensors that hand back some with their dimensions stored in reverse order and (C++; the Python form lets the
    library refuse them) some from a misaligned place in a buffer."""
    f, ins = _ops()[op]

    def run(order):
        args = [t.detach().clone().requires_grad_() for t in ins]
        if op == 'mixer':
            f.requires_grad_()
            args += list(f.parameters())
        count = iter(range(order, 1000))

        def unpack(t):
            i = next(count) % 3 if order else None
            if i == 0:
                return t.permute(*reversed(range(t.dim()))).contiguous().permute(*reversed(range(t.dim())))
            if i == 1 and form == 'c++':
                return th.cat([t.new_zeros(3), t.reshape(-1)])[3:].view(t.shape)
            return t

        with th.autograd.graph.saved_tensors_hooks(lambda t: t, unpack):
            out = f(*args[:len(ins)])
        return _grads(out if isinstance(out, (tuple, list)) else [out], args, 12)

    def compare():
        want = run(0)
        for order in (1, 2, 3):
            for a, b in zip(run(order), want, strict=True):
                _close(a, b, 1e-5 if op in ('ddlerp', 'expand_loras', 'mixer') else 0)  # sums over rows by atomics

    compare() if form == 'c++' else _python_form(monkeypatch, compare)


class _Sub(th.Tensor):
    seen = []

    @classmethod
    def __torch_function__(cls, func, types, args=(), kwargs=None):
        cls.seen.append(getattr(func, '__name__', ''))
        return super().__torch_function__(func, types, args, kwargs)


@pytest.mark.parametrize('op', ['attn', 'attn_ln', 'ddlerp', 'expand_loras', 'mixer'])
def test_subclasses(op, monkeypatch):
    """Subclasses of Tensor see the operators of the Python form, and outputs have the classes that it gives them."""
    f, ins = _ops()[op]
    for i in (0, len(ins) - 1):
        args = [t.as_subclass(_Sub) if j == i else t for j, t in enumerate(ins)]

        def run():
            _Sub.seen.clear()
            with th.no_grad():
                out = f(*args)
            return [type(o) for o in (out if isinstance(out, (tuple, list)) else [out])], list(_Sub.seen)

        got, want = run(), _python_form(monkeypatch, run)
        assert got == want and want[1]


@pytest.mark.filterwarnings('ignore')
@pytest.mark.parametrize('op', ['attn', 'attn_ln', 'ddlerp', 'expand_loras', 'mixer'])
def test_jit_trace_replays_on_other_inputs(op):
    f, ins = _ops()[op]
    other = [t.flip(0).contiguous() if t.dim() > 2 else t for t in ins]
    with th.no_grad():
        traced = th.jit.trace(f, tuple(ins), check_trace=False)
        got, want = traced(*other), f(*other)
    for a, b in zip(*[o if isinstance(o, (tuple, list)) else [o] for o in (got, want)], strict=True):
        assert not th.equal(b, th.zeros_like(b))
        _close(a, b, 2e-2 if op == 'mixer' else 0)  # (the traced layer is the Python form, see test_mixer)


def test_cast():
    from wind_rwkv.rwkv7 import _lib
    import ctypes
    sizes = [8, 24, 2048, 100000, 8]
    src = [th.randn(n, device='cuda') for n in sizes[:3]] + [th.randn(n, device='cuda').bfloat16() for n in sizes[3:]]
    kind = [0, 2, 0, 1, 1]
    dst = [th.empty(n, device='cuda', dtype=th.bfloat16 if k == 0 else th.float32) for n, k in zip(sizes, kind)]
    arr = lambda t, v: (t * len(v))(*v)
    n = len(sizes)
    rc = _lib.lib().wkv7_cast(arr(ctypes.c_void_p, [t.data_ptr() for t in src]), arr(ctypes.c_void_p, [t.data_ptr() for t in dst]), arr(ctypes.c_int64, sizes),
                              arr(ctypes.c_int, kind), n, th.cuda.current_stream().cuda_stream)
    assert rc == 0
    for s, d in zip(src, dst):
        assert th.equal(s.to(d.dtype), d)
    assert _lib.lib().wkv7_cast(None, None, None, None, 33, None) != 0


@pytest.mark.parametrize('M', [1, 130])
def test_proj_group(M):
    """Products of different widths in one launch: tiles that some of them do not have."""
    import ctypes
    from wind_rwkv.rwkv7 import _lib, proj
    K, widths, tanh = 72, [8, 136, 96], [(0, 8), (0, 0), (0, 64)]
    x = [th.randn(M, K, device='cuda').bfloat16() for _ in widths]
    w = [(th.randn(n, K, device='cuda') / 8).bfloat16() for n in widths]
    out = [th.empty(M, n, device='cuda', dtype=th.bfloat16) for n in widths]
    ptrs = lambda ts: (ctypes.c_void_p * 3)(*[t.data_ptr() for t in ts])
    ints = lambda v: (ctypes.c_int64 * 3)(*v)
    assert _lib.lib().wkv7_proj_gemm_group(3, ptrs(x), ptrs(w), ptrs(out), ints(widths), ints([f for f, _ in tanh]), ints([t for _, t in tanh]), M, K,
                                           th.cuda.current_stream().cuda_stream) == 0
    for a, b, o, t in zip(x, w, out, tanh):
        assert th.equal(proj(a, b, t), o)
    assert _lib.lib().wkv7_proj_gemm_group(5, None, None, None, None, None, None, M, K, None) != 0


@pytest.mark.parametrize('M', [1, 130])
def test_proj_group_of_several_widths_and_depths(M):
    """Products of different K in one launch, rows of A that are columns of a wider tensor: one K block and several, whole and partial."""
    import ctypes
    from wind_rwkv.rwkv7 import _lib, proj
    shapes, ld = [(8, 8), (264, 72), (96, 64), (128, 200), (16, 64), (40, 512)], [8, 72, 96, 208, 64, 520]
    x = [th.randn(M, s, device='cuda').bfloat16()[:, :k] for (_, k), s in zip(shapes, ld)]
    w = [(th.randn(n, k, device='cuda') / 8).bfloat16() for n, k in shapes]
    out = [th.empty(M, n, device='cuda', dtype=th.bfloat16) for n, _ in shapes]
    ptrs = lambda ts: (ctypes.c_void_p * 6)(*[t.data_ptr() for t in ts])
    ints = lambda v: (ctypes.c_int64 * 6)(*v)
    call = lambda count, k, lda: _lib.lib().wkv7_proj_gemm_group_ld(
        count, ptrs(x), ptrs(w), ptrs(out), ints([n for n, _ in shapes]), ints(k), ints(lda), ints([0] * 6), ints([0] * 6), M, th.cuda.current_stream().cuda_stream)
    ks = [k for _, k in shapes]
    assert call(6, ks, ld) == 0
    for a, b, o in zip(x, w, out):
        assert th.equal(proj(a.contiguous(), b), o)
    assert call(7, ks, ld) != 0 and call(6, ks, [k - 8 for k in ks]) != 0 and call(6, ks, [k + 4 for k in ld]) != 0


@pytest.mark.parametrize('B,T,C', [(1, 1, 64), (1, 130, 512), (1, 515, 2048), (2, 1200, 2048)])
def test_mixer_projections_of_few_rows(B, T, C, monkeypatch):
    """The layer on both sides of the lines between this library's and the framework's projections, against the Python form (the ops one
    by one): the bound of the layer's other tests."""
    from collections import namedtuple
    from wind_rwkv.rwkv7 import TimeMixer
    th.manual_seed(T)
    m = TimeMixer(namedtuple('Config', ['n_layer', 'n_head', 'n_embd'])(12, C // 64, C), 3).cuda()
    with th.no_grad():
        for p in m.parameters():
            p.add_(th.randn_like(p) * 0.02)
    x = th.randn(B, T, C, device='cuda').bfloat16()
    with th.no_grad():
        _close(m(x), _python_form(monkeypatch, lambda: m(x)), 1e-2)
