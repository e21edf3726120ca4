"""A grouped tensor-core launch whose pipeline waits run out (a limit of one poll; nothing
faults: the loads land, the products finish, the kernel returns) fails the call that
advanced the group, whichever geometry's tile gave up, and leaves no error behind for
later calls at the default limit.
"""
import numpy as np
import pytest

from plasmonx_b200 import _lib, configs
from plasmonx_b200.solver import Batch, Context, Solver

pytestmark = pytest.mark.gpu


def test_a_grouped_time_out_fails_the_step_and_is_reported_once():
    probs = [configs.na_sphere(radius=9.0, n_freq=5), configs.ag_sphere(radius=8.0, n_freq=5),
             configs.particle('Au', 'rod', 6.0, n_freq=5)]
    c = Context(0)
    solvers = [Solver(p, ctx=c, store_t=True) for p in probs]

    def batches():
        bs = [Batch(s, precision='mixed_bf16x3') for s in solvers]
        for k, (b, p) in enumerate(zip(bs, probs)):
            b.add(k, p.freqs, p.alpha_w, pol_mask=1, tol=1e-10)
        return bs

    def finish(bs):
        while any(b.active for b in bs):
            Batch.step_group([b for b in bs if b.active])
        out = [b.take(k)['results'] for k, b in enumerate(bs)]
        for b in bs:
            b.close()
        return out

    try:
        ref = finish(batches())
        for live in ([0, 1, 2], [0, 2]):
            bs = batches()
            c.set_wait_limit(1)
            with pytest.raises(_lib.PlxError) as e:
                Batch.step_group([bs[k] for k in live])
            assert e.value.code == 2 and 'timed out' in str(e.value)
            c.set_wait_limit(0)
            for b in bs:
                b.close()
            for s in solvers:                          # no geometry reports it a second time
                s.contract(np.ones((2, s.n_var)), 'bf16x3')
            for a, b in zip(finish(batches()), ref):
                np.testing.assert_array_equal(a, b)
    finally:
        for s in solvers:
            s.close()
        c.close()
