"""Host-side checks of the C ABI that need no GPU: the shared library loads, exports every
symbol include/wkv7_sm100.h declares, and rejects bad arguments before touching CUDA."""
import ctypes
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope='module')
def lib():
    import __graft_entry__ as ge
    ge.build()
    from wind_rwkv.rwkv7 import _lib
    return _lib.lib()


def declared_symbols():
    text = open(os.path.join(ROOT, 'include', 'wkv7_sm100.h')).read()
    text = re.sub(r'/\*.*?\*/', '', text, flags=re.S)
    return sorted(set(re.findall(r'\b(wkv7_[a-z0-9_]+)\s*\(', text)))


def test_header_symbols_are_exported_and_bound(lib):
    from wind_rwkv.rwkv7 import _lib
    names = declared_symbols()
    assert 'wkv7_fwd' in names and 'wkv7_bwd' in names
    for n in names:
        assert hasattr(lib, n), f'{n} declared in the header but not exported'
    assert sorted(_lib.exported_symbols()) == names, 'ctypes signatures out of sync with the header'


def test_status_strings(lib):
    assert lib.wkv7_status_string(0) == b'ok'
    for code in range(-9, 0):
        assert lib.wkv7_status_string(code) not in (b'', b'unknown status')
    assert lib.wkv7_status_string(-99) == b'unknown status'


def test_checkpoint_bytes(lib):
    assert lib.wkv7_checkpoint_bytes(64, 1024, 12, 64) == 64 * 12 * 64 * (64 * 64 + 4 * 16 * 16) * 4
    assert lib.wkv7_checkpoint_bytes(1, 64, 1, 32) == 0  # only N == 64 is built
    assert lib.wkv7_checkpoint_bytes(1, 0, 1, 64) == 0
    assert lib.wkv7_checkpoint_bytes(1, 17, 1, 64) == 2 * (64 * 64 + 4 * 16 * 16) * 4  # a partial last chunk has a record


def _fwd(lib, T=16, N=64, st=(1024, 64, 64), dtype=0, p=0x1000):
    return lib.wkv7_fwd(p, p, p, p, p, p, None, p, None, None, 1, T, 1, N, st[0], st[1], st[2], dtype, None)


def test_validation_happens_before_any_launch(lib):
    # none of these reach CUDA: the status comes from host-side checks alone
    assert _fwd(lib, T=1 << 40) == -8              # more checkpoint records than 32-bit row coordinates reach
    assert _fwd(lib, N=32) == -2                   # head size
    assert _fwd(lib, dtype=7) == -5                # dtype
    assert _fwd(lib, st=(1024, 60, 64)) == -4      # stride breaks 16-byte rows
    assert _fwd(lib, p=0x1004) == -4               # misaligned pointer
    assert _fwd(lib, T=-16) == -1
    assert _fwd(lib, st=(1024, 0, 64)) == -1       # 16 time steps in one place
    p = 0x1000
    for f, n in ((lib.wkv7_fwd, 10), (lib.wkv7_step, 9)):
        for strides in ((0, 128, 64), (2048, 128, 0)):  # two batch entries, two heads
            assert f(*([p] * n), 2, 16, 2, 64, *strides, 0, None) == -1
    assert lib.wkv7_fwd(None, None, None, None, None, None, None, None, None, None,
                        1, 16, 1, 64, 1024, 64, 64, 0, None) == -6
    # empty problems succeed without a launch
    assert lib.wkv7_fwd(None, None, None, None, None, None, None, None, None, None,
                        0, 16, 4, 64, 1024, 64, 64, 0, None) == 0
    # backward: dsT without sT
    p = 0x1000
    assert lib.wkv7_bwd(p, p, p, p, p, p, p, p, p, None, p, p, p, p, p, p, None,
                        1, 16, 1, 64, 1024, 64, 64, 0, None) == -6


def test_python_ops_refuse_cpu_tensors(lib):
    import torch as th
    from wind_rwkv.rwkv7 import attn
    x = th.zeros(1, 16, 64, dtype=th.bfloat16)
    with pytest.raises(RuntimeError, match='CUDA'):
        attn(x, x, x, x, x, x, 64)


def test_launchers_need_all_tensors_on_one_cuda_device(lib):
    """The wrappers make the tensors' device current for the launch and refuse mixed devices (a kernel launched on
    the current device with another device's pointers would fail or touch the wrong memory)."""
    import torch as th
    from wind_rwkv.rwkv7 import _lib
    with pytest.raises(RuntimeError, match='one device'):
        _lib.on_device(th.zeros(1), th.zeros(1, device='meta'))
    with pytest.raises(RuntimeError, match='CUDA'):
        _lib.on_device(th.zeros(1), None)


def test_status_word_is_readable_without_a_device(lib):
    """wkv7_peek_status is a host load of a managed variable; without a GPU it reports a launch error rather than
    crashing."""
    assert lib.wkv7_peek_status() in (0, -7)


def test_layouts_that_share_memory_are_told_apart():
    import torch as th
    from wind_rwkv.rwkv7.rwkv7_attn import _apart
    t = th.zeros(4096)
    for size, stride, want in [((3, 4, 2, 8), (64, 16, 8, 1), True), ((3, 4, 2, 8), (32, 16, 8, 1), False), ((3, 4, 2, 8), (0, 16, 8, 1), False),
                               ((3, 4, 2, 8), (16, 48, 8, 1), True), ((1, 4, 2, 8), (0, 16, 8, 1), True), ((3, 1, 2, 8), (16, 1, 8, 1), True),
                               ((3, 4, 2, 8), (128, 32, 8, 1), True), ((3, 4, 2, 8), (64, 16, 4, 1), False)]:
        assert _apart(t.as_strided(size, stride)) is want, (size, stride)


def test_backward_scratch_is_bounded(lib):
    """Tiles of the walked state gradients take 512 MB at most, whatever the number of chains and chunks, and a chain's tile of 18 KB a
    chunk comes in passes of 11 chunks or whole sequences."""
    flags, tile = lib.wkv7_workspace_bytes(), 64 * 72 * 4
    for chains in [1, 12, 149, 2000, 2647, 2648, 4096, 14563, 14564, 29127, 29128, 100000, 1 << 20]:
        for chunks in [1, 3, 4, 5, 10, 11, 12, 25, 300]:
            for B, H in ((chains, 1), (1, chains)):
                n = lib.wkv7_bwd_ws_bytes(B, 16 * chunks, H, 64, 1) - flags
                assert 0 <= n <= 512 << 20 and n % (chains * tile) == 0, (chains, chunks)
                per_pass = n // (chains * tile)
                assert per_pass == 0 or min(chunks, 11) <= per_pass <= chunks, (chains, chunks)
                assert per_pass or chunks < 4 or chains > 2647, (chains, chunks)
