"""Chains cut at the boundaries of equal shares of work (the *_ws entry points) against the same kernels with whole chains:
bit for bit the same, at chain counts around the number of resident CTAs and at the shortest and ragged lengths.  Few chains: the
backward's state gradient (attn) walked ahead of the rest by a kernel of its own, from 4 chunks on, in several passes where the
tiles would take more than 512 MB (12 chains of 2432 chunks: 2427 and 5)."""
import pytest
import torch as th

pytestmark = pytest.mark.gpu
N = 64


def sms():
    return th.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize('ln', [False, True])
@pytest.mark.parametrize('ckpt', [False, True])
@pytest.mark.parametrize('extra,T', [(1, 16), (1, 80), (-1, 48), (70, 7), (70, 33), (149, 1000), (400, 65)])
def test_forward(extra, T, ckpt, ln):
    forward_both_ways(extra, T, ckpt, ln)


@pytest.mark.parametrize('impl', [2, 3, 4, -4])
@pytest.mark.parametrize('ln', [False, True])
@pytest.mark.parametrize('T', [7, 16, 17, 33, 49, 64, 81, 96])
def test_forward_many_short_chains(T, ln, impl):
    """Some 17 chains of one to six chunks a CTA: a new start state every few chunks, written over the one before it when its last product has
    read it; slots, descriptors and state buffers all go round several times, and the cut chains' pieces have all lengths."""
    from wind_rwkv.rwkv7 import _lib
    old = _lib.set_fwd_impl(impl)
    try:
        forward_both_ways(2400, T, impl != -4, ln)
    finally:
        _lib.set_fwd_impl(old)


def forward_both_ways(extra, T, ckpt, ln):
    from wind_rwkv.rwkv7 import _lib, synthetic
    L = _lib.lib()
    B, H = 1, sms() + extra
    d = synthetic.wkv7_inputs(B, T, H, N, seed=T, dtype=th.bfloat16, device='cuda', s0_std=0.1)
    g, params = synthetic.attn_ln_extras(B, T, H, N, seed=T, dtype=th.bfloat16, device='cuda')
    ws = th.full((L.wkv7_workspace_bytes(),), 255, dtype=th.uint8, device='cuda')
    st = (T * H * N, H * N, N)

    def call(split):
        y, sT = th.full_like(d['r'], float('nan')), th.full((B, H, N, N), float('nan'), device='cuda')
        ck = th.zeros(L.wkv7_checkpoint_bytes(B, T, H, N) // 4 if ckpt else 4, device='cuda')
        a = [d[n].data_ptr() for n in 'rwkvab'] + ([g.data_ptr(), params.data_ptr()] if ln else [])
        a += [d['s0'].data_ptr(), y.data_ptr(), sT.data_ptr(), ck.data_ptr() if ckpt else None] + ([64e-5] if ln else [])
        a += [B, T, H, N, *st, 0] + ([ws.data_ptr()] if split else []) + [None]
        f = getattr(L, ('wkv7_attn_ln_fwd' if ln else 'wkv7_fwd') + ('_ws' if split else ''))
        assert f(*a) == 0
        th.cuda.synchronize()
        return y, sT, ck

    for a, b in zip(call(False), call(True)):
        assert bool(th.isfinite(a.float()).all()) and th.equal(a, b)
    assert L.wkv7_device_status() == 0


@pytest.mark.parametrize('ln', [False, True])
@pytest.mark.parametrize('extra,T,dsT', [(1, 16, False), (-1, 48, True), (70, 7, True), (200, 33, False), (149, 500, True), (400, 65, True),
                                         (-50, 64, True), (-49, 64, True), (-147, 48, True), (-147, 49, True), (-147, 2000, False), (-100, 1003, True), (-75, 333, True), (-136, 38900, True)])
def test_backward(extra, T, dsT, ln):
    from wind_rwkv.rwkv7 import _lib, synthetic
    from wind_rwkv.rwkv7.rwkv7_attn import fw_attn
    L = _lib.lib()
    B, H = 1, sms() + extra
    d = synthetic.wkv7_inputs(B, T, H, N, seed=T, dtype=th.bfloat16, device='cuda', s0_std=0.1)
    g, params = synthetic.attn_ln_extras(B, T, H, N, seed=T, dtype=th.bfloat16, device='cuda')
    _, sT, ck = fw_attn(*[d[n].view(B, T, H, N) for n in 'wrkvab'], d['s0'])
    gs = th.randn(B, H, N, N, device='cuda') if dsT else None
    ws = th.full(((L.wkv7_attn_ln_bwd_ws_bytes if ln else L.wkv7_bwd_ws_bytes)(B, T, H, N, 0),), 255, dtype=th.uint8, device='cuda')
    part = th.empty(B, 3, H * N, device='cuda')

    def call(split):
        outs = [th.full_like(d['r'], float('nan')) for _ in range(7 if ln else 6)]
        outs += [th.full((B, H, N, N), float('nan'), device='cuda')] + ([th.full_like(params, float('nan'))] if ln else [])
        a = [d[n].data_ptr() for n in 'rwkvab'] + ([g.data_ptr(), params.data_ptr()] if ln else [])
        a += [d['dy'].data_ptr(), ck.data_ptr(), _lib.ptr(gs), _lib.ptr(sT if dsT else None)]
        if ln:
            a += [o.data_ptr() for o in outs[:7]] + [outs[8].data_ptr(), part.data_ptr(), outs[7].data_ptr(), 64e-5]
        else:
            a += [o.data_ptr() for o in outs]
        a += [B, T, H, N, T * H * N, H * N, N, 0] + ([ws.data_ptr()] if split else []) + [None]
        assert getattr(L, ('wkv7_attn_ln_bwd' if ln else 'wkv7_bwd') + ('_ws' if split else ''))(*a) == 0
        th.cuda.synchronize()
        return outs

    for i, (a, b) in enumerate(zip(call(False), call(True))):
        assert bool(th.isfinite(a.float()).all())
        if i == 8:  # parameter gradients of a cut chain are summed in two pieces
            assert (a - b).norm() <= 1e-5 * a.norm()
        else:
            assert th.equal(a, b)
    assert L.wkv7_device_status() == 0


@pytest.mark.parametrize('chains,T,dsT', [(1, 48, True), (1, 49, False), (1, 64, True), (5, 100, True), (149, 49, True), (300, 65, False), (12, 38900, True)])
def test_backward_f32_walked(chains, T, dsT):
    """fp32 tensors: the state gradient walked by a kernel of its own (from four chunks on, in several passes where the tiles would take more
    than 512 MB), then all chunks in parallel, against the one-kernel form of the entry point without scratch.
    The same products to 2^-22 each, summed in another order: 1e-5 of the norm."""
    assert backward_f32_both_ways(chains, T, dsT) == (T > 48)


def backward_f32_both_ways(chains, T, dsT):
    """Compares the two; whether the scratch had room for tiles."""
    from wind_rwkv.rwkv7 import _lib, synthetic
    from wind_rwkv.rwkv7.rwkv7_attn import fw_attn
    L = _lib.lib()
    B, H = 1, chains
    d = synthetic.wkv7_inputs(B, T, H, N, seed=T, dtype=th.float32, device='cuda', s0_std=0.1)
    _, sT, ck = fw_attn(*[d[n].view(B, T, H, N) for n in 'wrkvab'], d['s0'])
    gs = th.randn(B, H, N, N, device='cuda') if dsT else None
    ws = th.full((L.wkv7_bwd_ws_bytes(B, T, H, N, 1),), 255, dtype=th.uint8, device='cuda')

    def call(walk):
        outs = [th.full_like(d['r'], float('nan')) for _ in range(6)] + [th.full((B, H, N, N), float('nan'), device='cuda')]
        a = [d[n].data_ptr() for n in 'rwkvab'] + [d['dy'].data_ptr(), ck.data_ptr(), _lib.ptr(gs), _lib.ptr(sT if dsT else None)]
        a += [o.data_ptr() for o in outs] + [B, T, H, N, T * H * N, H * N, N, 1] + ([ws.data_ptr()] if walk else []) + [None]
        assert getattr(L, 'wkv7_bwd' + ('_ws' if walk else ''))(*a) == 0
        th.cuda.synchronize()
        return outs

    for a, b in zip(call(False), call(True)):
        assert bool(th.isfinite(a).all()) and (a - b).norm() <= 1e-5 * a.norm()
    assert L.wkv7_device_status() == 0
    return ws.numel() > L.wkv7_workspace_bytes()


@pytest.mark.parametrize('chains,T', [(2647, 11 * 16), (2647, 12 * 16 + 5), (2648, 12 * 16)])
def test_backward_f32_walked_many_chains(chains, T):
    """As above where the tiles' 512 MB hold 11 chunks of every chain: one pass, two (11 chunks and 2), and one chain more, which is not
    walked and then has no scratch but the flags."""
    assert backward_f32_both_ways(chains, T, True) == (chains == 2647)


@pytest.mark.parametrize('form', ['c++', 'python'])
def test_backward_scratch_of_few_chains(form, monkeypatch):
    """The tiles of the walked state gradients are asked for where they are used (attn), not by attn_ln, which is not walked."""
    from wind_rwkv.rwkv7 import _lib, attn, attn_ln, synthetic
    if form == 'python':
        _lib.ext()
        monkeypatch.setattr(_lib, '_ext', type('Nothing', (), {'__getattr__': lambda self, name: lambda *a: None})())
    L = _lib.lib()
    B, T, H = 1, 4096, 12
    tiles = B * H * (T // 16) * 64 * 72 * 4
    assert L.wkv7_bwd_ws_bytes(B, T, H, N, 0) == L.wkv7_workspace_bytes() + tiles
    assert L.wkv7_attn_ln_bwd_ws_bytes(B, T, H, N, 0) == L.wkv7_workspace_bytes()
    d = synthetic.wkv7_inputs(B, T, H, N, seed=1, dtype=th.bfloat16, device='cuda')
    ins = [d[n].requires_grad_() for n in 'rwkvab']
    g, params = [x.requires_grad_() for x in synthetic.attn_ln_extras(B, T, H, N, seed=1, dtype=th.bfloat16, device='cuda')]
    for y, wrt in ((attn_ln(*ins, g, params, N), ins + [g, params]), (attn(*ins, N), ins)):
        th.cuda.synchronize()
        th.cuda.reset_peak_memory_stats()
        before = th.cuda.memory_stats()['requested_bytes.all.current']  # (as asked for: cached blocks are handed out up to 1 MB larger)
        grads = th.autograd.grad(y, wrt, d['dy'])
        extra = th.cuda.memory_stats()['requested_bytes.all.peak'] - before - sum(x.numel() * x.element_size() for x in grads)
        assert extra < tiles // 8 if len(wrt) == 8 else extra >= tiles  # (attn_ln's rest: ds0, partial sums)
        del grads


@pytest.mark.parametrize('form', ['c++', 'python'])
@pytest.mark.parametrize('dtype', [th.bfloat16, th.float32])
def test_backward_without_room_for_the_scratch(dtype, form, monkeypatch):
    """Where the tiles of the walked state gradients cannot be allocated, but the gradients can, the backward takes its one-kernel form:
    bf16 bit for bit the same, fp32 as in test_backward_f32_walked."""
    from wind_rwkv.rwkv7 import _lib, attn, synthetic
    if form == 'python':
        _lib.ext()
        monkeypatch.setattr(_lib, '_ext', type('Nothing', (), {'__getattr__': lambda self, name: lambda *a: None})())
    B, T, H = 1, 16384, 12
    tiles = _lib.lib().wkv7_bwd_ws_bytes(B, T, H, N, _lib.io_dtype(th.empty(0, dtype=dtype)))
    d = synthetic.wkv7_inputs(B, T, H, N, seed=1, dtype=dtype, device='cuda')
    ins = [d[n].requires_grad_() for n in 'rwkvab']
    y = attn(*ins, N)

    def limit(reserved):
        th.cuda.set_per_process_memory_fraction(min(1.0, reserved / th.cuda.get_device_properties(0).total_memory))

    try:
        th.cuda.synchronize()
        th.cuda.empty_cache()
        limit(th.cuda.memory_reserved())
        holes = []  # what other tests' remains leave free of the memory that the process keeps
        with pytest.raises(th.OutOfMemoryError):
            while True:
                holes.append(th.empty(tiles, dtype=th.uint8, device='cuda'))
        limit(float('inf'))
        want = th.autograd.grad(y, ins, d['dy'], retain_graph=True)
        held = th.cuda.memory_reserved()  # with all that one backward allocates, the tiles last
        want = [x.cpu() for x in want]
        th.cuda.empty_cache()
        asked = th.cuda.memory_stats()['num_ooms']
        limit(held - tiles // 2)
        got = [x.cpu() for x in th.autograd.grad(y, ins, d['dy'])]
    finally:
        limit(float('inf'))
    assert th.cuda.memory_stats()['num_ooms'] == asked + 1
    for a, b in zip(got, want):
        assert th.equal(a, b) if dtype == th.bfloat16 else (a - b).norm() <= 1e-5 * b.norm()
    assert _lib.lib().wkv7_device_status() == 0


@pytest.mark.parametrize('B,T,H,nseg', [(1, 34, 2, 2), (1, 3, 1, 3), (2, 99, 2, 3), (1, 256, 5, 16), (3, 1024, 7, 8)])
@pytest.mark.parametrize('s0', [False, True])
def test_time_split(B, T, H, nseg, s0):
    """Sequences cut into parallel segments: one and several sequences, ragged segments, against the uncut forward."""
    from wind_rwkv.rwkv7 import _lib, attn, synthetic
    d = synthetic.wkv7_inputs(B, T, H, N, seed=T, dtype=th.bfloat16, device='cuda', s0_std=0.1)
    ins, s = [d[n] for n in 'rwkvab'], d['s0'] if s0 else None
    with th.no_grad():
        want = attn(*ins, N, s0=s, return_state=True)
        got = attn(*ins, N, s0=s, return_state=True, time_split=nseg)
    for a, b in zip(got, want):
        assert a.dtype == b.dtype and (a.float() - b.float()).norm() <= 4e-3 * b.float().norm()
    assert _lib.lib().wkv7_device_status() == 0


@pytest.mark.parametrize('B,T,H', [(1, 1024, 12), (1, 1008, 12), (2, 1024, 12), (1, 1008, 2)])
def test_time_split_maps_of_cut_chains(B, T, H):
    """The segments' maps where they matter (slow decays, start states of size 1) and where CTAs hand half-walked ones on (180 and 384
    segments on 148 SMs, whole and partial last chunks), against the uncut forward.  M's products are single TF32 like the uncut
    call's: the bound is that of test_time_split."""
    from wind_rwkv.rwkv7 import _lib, attn, synthetic
    d = synthetic.wkv7_inputs(B, T, H, N, seed=T + B, dtype=th.bfloat16, device='cuda', s0_std=1.0)
    d['w'] = (d['w'].float() * 0.5 - 5.7).bfloat16()
    ins = [d[n] for n in 'rwkvab']
    with th.no_grad():
        want = attn(*ins, N, s0=d['s0'], return_state=True)
        got = attn(*ins, N, s0=d['s0'], return_state=True, time_split=16)
    for a, b in zip(got, want):
        assert (a.float() - b.float()).norm() <= 4e-3 * b.float().norm()
    assert _lib.lib().wkv7_device_status() == 0


@pytest.mark.parametrize('chains,T,s0', [(1, 1, False), (1, 16, True), (2, 17, True), (3, 48, False), (5, 100, True), (148, 65, True), (149, 500, True), (150, 33, False)])
def test_forward_f32(chains, T, s0):
    """fp32 forward on both sides of the line between its two kernels, against a float64 recurrence on the CPU: fewer chunks than preparation
    groups, partial last chunks, as many chains as SMs and more.  1e-5 of the norm: fp32 sums of products that are right to 2^-22."""
    from wind_rwkv.rwkv7 import _lib, attn, synthetic
    d = synthetic.wkv7_inputs(1, T, chains, N, seed=T, dtype=th.float32, device='cuda', s0_std=0.1)
    y, sT = attn(*[d[n] for n in 'rwkvab'], N, s0=d['s0'] if s0 else None, return_state=True)
    r, w, k, v, a, b = [d[n].view(T, chains, N).double().cpu() for n in 'rwkvab']
    S = d['s0'][0].double().cpu() if s0 else th.zeros(chains, N, N, dtype=th.float64)
    ref = []
    for t in range(T):
        sa = S @ a[t].unsqueeze(-1)
        S = S * th.exp(-th.exp(w[t])).unsqueeze(1) + sa @ b[t].unsqueeze(1) + v[t].unsqueeze(-1) @ k[t].unsqueeze(1)
        ref.append((S @ r[t].unsqueeze(-1)).squeeze(-1))
    for got, want in ((y.view(T, chains, N), th.stack(ref)), (sT[0], S)):
        assert (got.double().cpu() - want).norm() <= 1e-5 * want.norm()
    assert _lib.lib().wkv7_device_status() == 0
