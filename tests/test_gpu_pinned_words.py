"""Where a solve's steps leave their residuals: pinned host memory, or device memory and a
copy where the system pins none.  A fake of cudaHostAlloc, preloaded into a child process,
counts the calls and refuses all of them, or the first ones, on request; the solves' bits
are the same in every case.
"""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

FAKE = r'''
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stdlib.h>
static int calls = 0;
int fake_calls(void) { return calls; }
int cudaHostAlloc(void **p, size_t n, unsigned flags) {
    ++calls;
    const char *refuse = getenv("REFUSE_PINNED");      /* that many calls */
    if (refuse && calls <= atoi(refuse)) return 2;     /* cudaErrorMemoryAllocation */
    void *rt = dlopen("libcudart.so.12", RTLD_NOLOAD | RTLD_LAZY);          /* the library's, loaded by now */
    int (*real)(void **, size_t, unsigned) = rt ? (int (*)(void **, size_t, unsigned))dlsym(rt, "cudaHostAlloc") : 0;
    return real ? real(p, n, flags) : 1;
}
'''

CHILD = r'''
import ctypes, hashlib, json, numpy as np
from plasmonx_b200 import _lib, configs
from plasmonx_b200.solver import Batch, Context, Solver
calls = ctypes.CDLL(None).fake_calls
out = {}
ctx = Context(0)
digest = lambda o: hashlib.sha256(o['x'].tobytes() + o['status'].tobytes()).hexdigest()
p = configs.na_sphere(radius=14.0, n_freq=9, method='iterative')
with Solver(p, ctx=ctx) as sv:
    tol = 1e-10 * float(np.linalg.norm(sv.rhs(0)[:, 0]))
    short = lambda: digest(sv.solve(pol_mask=1, tol=1e-2 * float(np.linalg.norm(sv.rhs(0)[:, 0])), max_krylov=40, want_x=True))
    out['short'] = short()
    full = [sv.solve(tol=tol, want_x=True) for _ in range(4)]
    out['full'] = [digest(o) for o in full]
    out['status'] = int(max(abs(o['status']).max() for o in full))
    out['short_again'] = short()
p = configs.ag_sphere(radius=9.0, n_freq=9, method='iterative')
with Solver(p, ctx=ctx) as sv:
    out['mixed'] = [digest(sv.solve(precision='mixed_bf16x3', want_x=True)) for _ in range(3)]
out['calls'] = calls()
ctx.close()
print(json.dumps(out))
'''


@pytest.fixture(scope='module')
def runs(tmp_path_factory):
    d = tmp_path_factory.mktemp('fake')
    src, lib = d / 'fake.c', d / 'fake.so'
    src.write_text(FAKE)
    subprocess.run(['gcc', '-shared', '-fPIC', '-o', str(lib), str(src), '-ldl'], check=True)
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    res = []
    for refuse in (0, 1000000, 2):
        env = dict(os.environ, LD_PRELOAD=str(lib), PYTHONPATH=root, REFUSE_PINNED=str(refuse))
        r = subprocess.run([sys.executable, '-c', CHILD], env=env, cwd=root, capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        res.append(json.loads(r.stdout.strip().splitlines()[-1]))
    return res


def test_a_context_keeps_the_blocks_it_pins(runs):
    """One, and a second one for the cycle of an inner solve that is set up before the
    cycle it follows is released."""
    assert 1 <= runs[0]['calls'] <= 2


def test_refused_pinned_memory_costs_copies_only(runs):
    """Refused for good, and for the first two tries (hundreds of steps apart)."""
    pinned, refused, late = runs
    assert refused['calls'] >= 3 and 3 <= late['calls'] <= 4
    for r in (refused, late):
        assert r['status'] == 0
        for key in ('short', 'short_again', 'full', 'mixed'):
            assert r[key] == pinned[key], key


def test_the_bits_do_not_depend_on_where_the_words_lie(runs):
    r = runs[0]
    assert r['short'] == r['short_again']
    assert len(set(r['full'])) == 1 and len(set(r['mixed'])) == 1
