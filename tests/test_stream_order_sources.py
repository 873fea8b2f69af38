"""Kernels that wait for the one ahead of them (stream_wait, stream_order) must not read anything before that.  The compiler may move loads
through __restrict__ pointers ahead of the wait, so each such parameter goes through after_stream_order behind it (read from the sources)."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'wind-rwkv7_b200', 'csrc')


def kernels():
    for name in sorted(os.listdir(CSRC)):
        text = open(os.path.join(CSRC, name)).read()
        for part in re.split(r'^(?:template.*\n)?__global__ ', text, flags=re.M)[1:]:
            head, _, body = part.partition(') {\n')
            yield name, head, re.split(r'^}', body, maxsplit=1, flags=re.M)[0]


def test_restrict_pointers_are_read_behind_the_wait():
    seen = 0
    for name, head, body in kernels():
        wait = re.search(r'stream_(order|wait)\(\);', body)
        if not wait:
            continue
        for param in re.findall(r'__restrict__ (\w+)', head):
            seen += 1
            assert re.search(rf'\b{param} = after_stream_order\({param}\)', body[wait.end():]), f'{name}: {head.split("(")[-2][-30:]}: {param}'
            assert not re.search(rf'\b{param}\b', body[:wait.start()]), f'{name}: {param} is used ahead of the wait'
    assert seen >= 15
