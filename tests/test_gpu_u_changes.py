"""A velocity that turns zero and back between the fused calls of one context, on boxes without the
Hall term, whose inflow data depends on the time: every call equals the same call of a fresh
context that starts from the same fields and the same time, so no velocity plane, flag or graph of
an earlier call is read."""
from __future__ import annotations

import numpy as np
import pytest

from tests.helpers import maps_for

pytestmark = pytest.mark.gpu


def _call(ctx, b, u, t, steps):
    dev = [ctx.vec(b), ctx.vec(), ctx.vec(), ctx.vec(), ctx.vec(u), ctx.scalar(np.ones(ctx.n_pad)), ctx.scalar(t, n=2)]
    ctx.time_steps(*dev, steps)
    return ctx.get_vec(dev[0]), ctx.get_vec(dev[1]), ctx.get_scalar(dev[6], n=2)


@pytest.mark.parametrize("dissipation", ["NONE", "FIRST_ORDER", "ADAPTIVE"])
@pytest.mark.parametrize("nodes", [(17, 13, 12), (18, 13, 12)])
@pytest.mark.parametrize("integrator", ["SSPRK33", "KennedyCarpenterLewis2R54C", "CarpenterKennedy2N54"])
def test_calls_that_change_u_equal_fresh_contexts_at_the_same_time(integrator, nodes, dissipation):
    c = dict(order=4, testcase="rotation_3D", nodes=nodes, lo=-1.0, hi=1.0, integrator=integrator, dt=1e-3,
             dissipation=dissipation)
    ctx = maps_for(c).context()
    rng = np.random.default_rng(3)
    b = rng.standard_normal((ctx.n_pad, 4)) * [1, 1, 1, 0]
    u1 = 0.3 * rng.standard_normal((ctx.n_pad, 4)) * [1, 1, 1, 0]
    zero, one = np.zeros_like(u1), np.zeros_like(u1)
    one[ctx.n - 1, 2] = 0.25
    t = np.zeros(2)
    # one set of the context's own arrays, so that its graphs are used again
    dev = [ctx.vec(b), ctx.vec(), ctx.vec(), ctx.vec(), ctx.vec(u1), ctx.scalar(np.ones(ctx.n_pad)), ctx.scalar(t, n=2)]
    for k, u in enumerate((u1, zero, one, zero, u1, u1, zero)):
        dev[4].upload(u)
        fresh = maps_for(c).context()
        want = _call(fresh, b, u, t, 1 + k % 3)
        fresh.close()
        ctx.time_steps(*dev, 1 + k % 3)
        b, t = ctx.get_vec(dev[0]), ctx.get_scalar(dev[6], n=2)
        np.testing.assert_array_equal(b, want[0])
        np.testing.assert_array_equal(ctx.get_vec(dev[1]), want[1])
        np.testing.assert_array_equal(t, want[2])
        if u is not zero:
            assert t[0] > 0
    ctx.close()
