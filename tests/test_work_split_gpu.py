"""Chains cut at the boundaries of equal shares of work (the *_ws entry points) against the same kernels with whole chains:
bit for bit the same, at chain counts around the number of resident CTAs and at the shortest and ragged lengths."""
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
