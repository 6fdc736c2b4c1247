"""Adaptive and first-order dissipation of the one-node column kernels where their paths change:
fields with a thin sheet in part of the grid, so that some warps hold kappas between the
thresholds, some above and some only zeros, on odd periodic grids, even ones and boxes, with a
compile-time and a run-time flux mask: one step against the oracle to 1e-12 of the field's
scale (the oracle evaluates every kappa)."""
from __future__ import annotations

import math

import numpy as np
import pytest

from oracle.hostloops import time_loop
from tests.helpers import field_ok, maps_for, oracle_for

pytestmark = pytest.mark.gpu

HP = 4.0 * math.pi / 3.0


@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("diss", ["ADAPTIVE", "FIRST_ORDER"])
@pytest.mark.parametrize("nodes, periodic", [((35, 17, 18), True), ((36, 16, 17), True), ((35, 17, 18), False)])
@pytest.mark.parametrize("order", [2, 4, 6])
def test_sheet_matches_oracle(order, nodes, periodic, diss, split):
    form = "SPLIT" if split else "CENTRAL"
    c = dict(order=order, testcase="hall_periodic" if periodic else "rotation_3D", nodes=nodes, lo=0.0 if periodic else -1.0,
             hi=HP if periodic else 1.0, periodic=periodic, hall=periodic, dissipation=diss,
             integrator="CarpenterKennedy2N54", dt=1e-3, uibj="SPLIT" if split else "PRODUCT", source=form, ujbi=form)
    o = oracle_for(c)
    b, u = o.vec(), o.vec()
    o.run("init_b", o.cfg.nodes, b)
    o.run("init_u", o.cfg.nodes, u)
    i = np.arange(o.N)
    x, z = i % nodes[0], i // (nodes[0] * nodes[1])
    b[:, 1] += np.where(z > nodes[2] // 2, 40.0, 2.0) * np.exp(-((x - 9.0) / 1.5) ** 2)   # a sheet, stronger above
    host = [b.copy(), o.vec(), o.vec(), o.vec(), u, o.scalar(fill=1.0), np.zeros(2)]
    time_loop(o, c["integrator"], c["hall"], False, 1, *host)
    ctx = maps_for(c).context()
    dev = [ctx.vec(b), ctx.vec(), ctx.vec(), ctx.vec(), ctx.vec(u), ctx.scalar(np.ones(ctx.n_pad)),
           ctx.scalar(np.zeros(2), n=2)]
    ctx.time_steps(*dev, 1)
    ok, e = field_ok(ctx.get_vec(dev[0]), host[0], 1e-12)
    assert ok, e
    ctx.close()
