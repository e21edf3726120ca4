"""A shared-memory array that kernels access through a wider vector type is declared with
that alignment: its element type alone guarantees less, and its place among a kernel's
other shared variables is the compiler's choice."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'plasmonx_b200', 'csrc')
BYTES = {'double2': 16, 'float4': 16, 'int4': 16, 'uint4': 16, 'float2': 8, 'int2': 8}
ELEMENT = {'double': 8, 'float': 4, 'int': 4, 'int32_t': 4, 'uint32_t': 4, 'uint8_t': 1}


@pytest.mark.parametrize('path', sorted(glob.glob(os.path.join(CSRC, '*.cu')) + glob.glob(os.path.join(CSRC, '*.cuh'))),
                         ids=os.path.basename)
def test_vector_access_to_shared_arrays(path):
    with open(path) as f:
        text = f.read()
    shared = {}
    for m in re.finditer(r'__shared__\s+(?:__align__\((\d+)\)\s+)?(\w+)\s+([^;]*);', text):
        for name in re.findall(r'(\w+)\s*\[', m.group(3)):
            shared[name] = max(int(m.group(1) or 0), ELEMENT.get(m.group(2), 0))
    for m in re.finditer(r'reinterpret_cast<(?:const )?(\w+) \*>\(&(\w+)\[', text):
        wide, name = m.groups()
        if wide in BYTES and shared.get(name):
            assert shared[name] >= BYTES[wide], '%s as %s' % (name, wide)
