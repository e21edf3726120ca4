"""The library's host code names no instruction of one host architecture outside the
header that chooses by architecture, and that header preprocesses to other hosts' forms."""
import glob
import os
import re
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'plasmonx_b200', 'csrc')
HEADER = os.path.join(CSRC, 'cpu_relax.h')
X86 = re.compile(r'__builtin_ia32_|\b_mm_\w+|[xei]mmintrin\.h')


def test_no_x86_builtin_in_the_sources():
    for path in glob.glob(os.path.join(CSRC, '*')):
        if os.path.isfile(path) and path != HEADER:
            with open(path) as f:
                assert not X86.search(f.read()), path


@pytest.mark.parametrize('flags,token', [([], '__builtin_ia32_pause'),
                                         (['-U__x86_64__', '-U__i386__', '-D__aarch64__'], 'yield'),
                                         (['-U__x86_64__', '-U__i386__', '-U__aarch64__'], None)])
def test_the_hint_by_architecture(flags, token):
    if not flags and os.uname().machine != 'x86_64':
        pytest.skip('an x86-64 host')
    text = subprocess.run(['g++', '-E', '-P', '-x', 'c++', *flags, HEADER], check=True, capture_output=True,
                          text=True).stdout
    assert bool(X86.search(text)) == (token == '__builtin_ia32_pause')
    assert ('yield' in text) == (token == 'yield')
