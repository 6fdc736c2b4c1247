"""Stage-by-stage sessions (ieq_stages_*) on boxes with odd rows, whose fused state has a row
pitch of nx + 1 outside a session and of nx inside one: fused calls, adjoint sweeps and batches
made before, during and after a session -- also one that ends with an error -- give what they give
on a context that never had one.  Every field is compared for equality."""
from __future__ import annotations

import numpy as np
import pytest

from inductioneq_b200.batch import Batch
from inductioneq_b200.lib import IeqError
from tests.helpers import maps_for

pytestmark = pytest.mark.gpu

CASES = {
    "rotation": dict(order=4, testcase="rotation_3D", nodes=(17, 13, 12), lo=-1.0, hi=1.0, integrator="SSPRK33",
                     dt=1e-3),
    "confined_hall": dict(order=4, testcase="confined_domain", nodes=(17, 13, 12), lo=0.0, hi=1.0, hall=True,
                          dissipation="HIGH_ORDER", integrator="CarpenterKennedy2N54", dt=1e-5),
}


class Run:
    """One context with its fields; `advance` returns what a fused call left in them."""

    def __init__(self, name):
        self.ctx = c = maps_for(CASES[name]).context()
        b, u = c.vec(), c.vec()
        c.kernel("init_b", b)
        c.kernel("init_u", u)
        bh = c.get_vec(b)
        bh[: c.n, :3] += 1e-2 * np.random.default_rng(3).standard_normal((c.n, 3))
        self.three = CASES[name]["integrator"] == "SSPRK33"
        self.f = [c.vec(bh), c.vec(), c.vec() if self.three else None, c.vec(), u,
                  c.scalar(np.linspace(0.8, 1.3, c.n_pad)), c.scalar(np.zeros(2), n=2)]
        self.s = [c.vec(bh), c.vec(), c.vec() if self.three else None, c.vec(), u]   # a session's own fields
        self.lam0 = np.random.default_rng(4).standard_normal((c.n_pad, 4))

    def advance(self, steps):
        self.ctx.time_steps(*self.f, steps)
        got = [self.ctx.get_vec(x) for x in self.f[:4] if x is not None]
        return got + [self.ctx.get_scalar(self.f[6], n=2)]

    def adjoint(self):
        lam = self.ctx.vec(self.lam0)
        self.ctx.adjoint_steps(self.f[0], lam, self.f[4], self.f[5], 3, 2)
        return [self.ctx.get_vec(lam)]

    def begin(self):
        return self.ctx.stages_begin(*self.s)

    def end(self):
        self.ctx.stages_end(*self.s, self.f[5])

    def failing_end(self):
        with pytest.raises(IeqError):
            self.ctx.stages_end(None, *self.s[1:], self.f[5])


def _same(a, b):
    for x, y in zip(a, b, strict=True):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("fails", [False, True])
def test_fused_calls_after_a_session(name, fails):
    a, ref = Run(name), Run(name)
    _same(a.advance(3), ref.advance(3))
    a.begin()
    a.failing_end() if fails else a.end()
    _same(a.advance(3), ref.advance(3))
    _same(a.adjoint(), ref.adjoint())
    a.ctx.close()
    ref.ctx.close()


@pytest.mark.parametrize("name", sorted(CASES))
def test_an_end_without_a_session_changes_nothing(name):
    a, ref = Run(name), Run(name)
    a.failing_end()
    with pytest.raises(IeqError):
        a.end()
    _same(a.advance(2), ref.advance(2))
    a.ctx.close()
    ref.ctx.close()


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("before", [False, True])
def test_fused_calls_within_a_session(name, before):
    # `before`: the graphs exist when the session begins; else the call inside captures them
    a, ref = Run(name), Run(name)
    if before:
        _same(a.advance(2), ref.advance(2))
        _same(a.adjoint(), ref.adjoint())
    a.begin()
    _same(a.advance(2), ref.advance(2))
    _same(a.adjoint(), ref.adjoint())
    a.end()
    _same(a.advance(2), ref.advance(2))
    _same(a.adjoint(), ref.adjoint())
    a.ctx.close()
    ref.ctx.close()


@pytest.mark.parametrize("mode", ["persistent", "stages", "branches"])
def test_batch_bound_within_a_session(mode):
    got = []
    for session in (False, True):
        bt = Batch([(13, 4, 0.7, 1e-3), (17, 6, 0.9, 1e-3)])
        bt.init()
        extra = [[c.vec() for _ in range(5)] for c in bt.ctxs]
        if session:
            for c, e in zip(bt.ctxs, extra):
                c.stages_begin(*e)
        bt.bind()
        if session:
            for c, e in zip(bt.ctxs, extra):
                c.stages_end(*e, c.scalar(np.ones(c.n_pad)))
        bt.run(2, mode=mode)
        bt.unbind()
        got.append([c.get_vec(f["b"]) for c, f in zip(bt.ctxs, bt.fields)])
        bt.close()
    _same(*got)
