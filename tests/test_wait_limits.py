"""The bounds of the device-side waits, read from the sources (no GPU: nothing here can be made to run out on purpose).  In the
tcgen05 forward one preparation group waits for the state of a cut chain while every other warp of the CTA stands still; their waits
must outlast that one, or the CTA reports a lost condition that is only late."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'wind-rwkv7_b200', 'csrc')


def _read(name):
    return open(os.path.join(CSRC, name)).read()


def _constants(text, known):
    for name, expr in re.findall(r'constexpr long long (\w*LIMIT) = ([^;]+);', text):
        known[name] = eval(re.sub(r'(\d)LL\b', r'\1', expr), {}, known)
    return known


def test_waits_that_span_a_handoff_outlast_it():
    common, fwd = _read('wkv7_common.cuh'), _read('wkv7_fwd_tc.cu')
    c = _constants(common, {})
    limit = re.search(r'void wait_handoff\(.*?clock64\(\) - start > ([\w *]+)\)', common, re.S).group(1)
    handoff = eval(limit, {}, c)
    c = _constants(fwd, c)
    assert 'wait_handoff(' in fwd
    # the kernel's waits all go through mbar_wait (default: WAIT_LIMIT) and the score warps' idle loop
    assert re.search(r'void mbar_wait\([^)]*long long limit = WAIT_LIMIT\)', fwd)
    assert re.search(r'clock\(\) - since > \(uint32_t\)WAIT_LIMIT\) give_up', fwd)
    assert handoff < c['WAIT_LIMIT'] < 1 << 32, 'counted in 32 bits'
    assert c['WAIT_LIMIT'] < 2 * 1_965_000_000, 'about a second at the highest clock'
