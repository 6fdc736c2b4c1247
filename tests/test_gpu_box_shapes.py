"""Boxes on the edges of the launch rules of the pair kernels: one round of blocks and more, rows
of whole 8-pair blocks and others, and the x boundary columns in their band beside odd rows (whose
last interior node goes with the band), against the same step with one node per thread.

Both sum every node's terms in one order; what differs is the compiler's choice of fused
multiply-adds.  A stage is a few hundred operations of relative 1.1e-16 (FP64) on terms up to a
few hundred times the result near the walls, two steps are 6 to 10 stages: 1e-12 of the scale.
"""
from __future__ import annotations

import numpy as np
import pytest

from tests.helpers import maps_for

pytestmark = pytest.mark.gpu

ROT = dict(testcase="rotation_3D", lo=-1.0, hi=1.0, integrator="SSPRK33")
CONF = dict(testcase="confined_domain", lo=0.0, hi=1.0, hall=True, integrator="CarpenterKennedy2N54")
CASES = [(dict(base, order=o, nodes=n, xband=band), dt)
         for base, dt in ((ROT, 2e-3), (CONF, 1e-6))
         for o, n in ((2, (5 + 12, 9, 10)), (2, (97, 20, 19)), (2, (98, 33, 34)), (4, (17, 18, 19)), (4, (50, 50, 50)),
                      (4, (91, 30, 31)), (4, (96, 40, 40)), (6, (21, 22, 23)), (6, (93, 25, 24)), (6, (64, 64, 33)))
         for band in (1, 2)]
CASES += [(dict(CONF, order=4, nodes=n, xband=2, dissipation="HIGH_ORDER"), 1e-6) for n in ((31, 17, 18), (32, 17, 18))]
CASES += [(dict(ROT, order=o, nodes=(33, 17, 18), xband=2, dissipation="FIRST_ORDER"), 2e-3) for o in (2, 4, 6)]
# adaptive dissipation: compact blocks from three rounds on, against blocks of 32-node rows
CASES += [(dict(base, order=o, nodes=n, xband=1, dissipation="ADAPTIVE"), dt)
          for base, dt in ((ROT, 2e-3), (CONF, 1e-6)) for o, n in ((2, (57, 66, 71)), (4, (97, 41, 67)), (6, (66, 65, 64)))]


def _run(c, dt, **kw):
    ctx = maps_for(dict(c, dt=dt, **kw)).context()
    b, b2, b3, cb, u = (ctx.vec() for _ in range(5))
    ctx.kernel("init_b", b)
    ctx.kernel("init_u", u)
    rng = np.random.default_rng(11)
    x = ctx.get_vec(b)
    x[: ctx.n, :3] += 0.1 * rng.standard_normal((ctx.n, 3))
    b = ctx.vec(x)
    rho = np.ones(ctx.n_pad)
    rho[: ctx.n] += 0.1 * rng.random(ctx.n)
    ctx.time_steps(b, b2, b3, cb, u, ctx.scalar(rho), ctx.scalar(np.zeros(2), n=2), 2)
    out = ctx.get_vec(b)[: ctx.n, :3].copy()
    ctx.close()
    return out


@pytest.mark.parametrize("c, dt", CASES)
def test_pair_launches_equal_one_node_per_thread(c, dt):
    ref = _run(dict(c, xband=0), dt, col_pairs=0, col_block=(32, 4, 1))
    got = _run(c, dt)
    assert np.isfinite(ref).all()
    assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max()
