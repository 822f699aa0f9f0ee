"""Frame kernels may begin before their predecessor has finished (programmatic
stream serialization), so what they read of global memory has to stay behind
their wait: the wait comes first, and no load and no pointer promises that the
memory is constant while the kernel runs. Read from the sources."""
import glob
import os
import re

import vk_order_independent_transparency_gb300 as oit

CSRC = os.path.join(os.path.dirname(os.path.abspath(oit.__file__)), 'csrc')


def sources():
    """{file name: its text without comments} of the files with frame kernels
    and the headers they include."""
    text = {}
    for path in glob.glob(os.path.join(CSRC, '*.cu')) + glob.glob(os.path.join(CSRC, '*.cuh')):
        with open(path) as f:
            s = re.sub(r'/\*.*?\*/', '', f.read(), flags=re.S)
        text[os.path.basename(path)] = re.sub(r'//[^\n]*', '', s)
    pending = [n for n, s in text.items() if 'launch_in_frame(' in s]
    out = {}
    while pending:
        n = pending.pop()
        if n in out or n not in text:
            continue
        out[n] = text[n]
        pending += re.findall(r'#include "([^"]+)"', text[n])
    return out


def test_frame_kernels_wait_first():
    src = sources()
    launched = set()
    for s in src.values():
        launched |= set(re.findall(r'launch_in_frame\(\s*(k_\w+)', s))
    assert len(launched) > 10
    every = '\n'.join(src.values())
    for k in launched:
        bodies = re.findall(r'__global__[^;{}]*?\b%s\s*\([^{;]*\)\s*\{\s*([^\n]*)' % k, every)
        assert bodies, k
        assert all(b.strip() == 'frame_order();' for b in bodies), (k, bodies)


def test_frame_memory_is_read_with_ordinary_loads():
    for name, s in sources().items():
        assert '__restrict__' not in s, name
        for load in re.findall(r'__ld(?:g|cg|cs|ca|lu|cv)\([^;]*', s):
            assert load.startswith('__ldg(&g_srgb.'), (name, load)
        # volatile: kept in order with the wait
        for asm in re.findall(r'asm\s*(\w*)\s*\(\s*"ld\.', s):
            assert asm == 'volatile', name
        assert 'ld.global.nc' not in s, name
