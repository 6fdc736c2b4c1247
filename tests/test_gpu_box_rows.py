"""The boundary-row paths of the box stage and curl kernels at the smallest boxes of every
operator (2 * NUM_BOUNDS nodes: no interior row in an axis) and one or two nodes above, where a
row's entries, the reach of a node pair along x and the two ends of an axis meet: one step
against the oracle, every field to 1e-12 of its own scale plus the forward-error floor of the
registers (tests/helpers.py)."""
from __future__ import annotations

import numpy as np
import pytest

from oracle.hostloops import time_loop
from tests.golden.cases import NOISE_SEED
from tests.helpers import field_ok, maps_for, oracle_for, rounding_floor

pytestmark = pytest.mark.gpu

NB = {(2, False): 1, (4, False): 4, (6, False): 6, (2, True): 3, (4, True): 6, (6, True): 8}
# testcase, integrator, hall, dissipation, flux forms (u_i B_j, source, u_j B_i)
RUNS = [("rotation_3D", "SSPRK33", False, "NONE", ("PRODUCT", "CENTRAL", "CENTRAL")),
        ("rotation_3D", "SSPRK33", False, "NONE", ("SPLIT", "SPLIT", "SPLIT")),
        ("rotation_3D", "SSPRK33", False, "HIGH_ORDER", ("PRODUCT", "CENTRAL", "CENTRAL")),
        ("confined_domain", "CarpenterKennedy2N54", True, "HIGH_ORDER", ("CENTRAL", "ZERO", "CENTRAL")),
        ("confined_domain", "CarpenterKennedy2N54", True, "FIRST_ORDER", ("PRODUCT", "CENTRAL", "CENTRAL"))]


@pytest.mark.parametrize("run", range(len(RUNS)))
@pytest.mark.parametrize("extra", [0, 1, 2])
@pytest.mark.parametrize("order, extended", sorted(NB))
def test_smallest_boxes_match_oracle(order, extended, extra, run):
    testcase, integrator, hall, diss, forms = RUNS[run]
    m = max(2 * NB[order, extended], 4)
    hall_dt = 1e-4
    c = dict(order=order, extended=extended, testcase=testcase, nodes=(m + extra, m + 1, m), lo=0.0 if hall else -1.0,
             hi=1.0, hall=hall, dissipation=diss, integrator=integrator, dt=hall_dt if hall else 5e-3,
             uibj=forms[0], source=forms[1], ujbi=forms[2])
    o = oracle_for(c)
    b, u = o.vec(), o.vec()
    o.run("init_b", o.cfg.nodes, b)
    o.run("init_u", o.cfg.nodes, u)
    b[:, :3] += 1e-2 * np.random.default_rng(NOISE_SEED).standard_normal((o.N, 3))
    host = [b.copy(), o.vec(), o.vec(), o.vec(), u, o.scalar(fill=1.0), np.zeros(2)]
    time_loop(o, integrator, hall, False, 1, *host)
    ctx = maps_for(c).context()
    dev = [ctx.vec(b), ctx.vec(), ctx.vec(), ctx.vec(), ctx.vec(u), ctx.scalar(np.ones(ctx.n_pad)),
           ctx.scalar(np.zeros(2), n=2)]
    ctx.time_steps(*dev, 1)
    mb, mu = float(np.abs(b).max()), float(np.abs(u).max())
    for i in ((0, 1, 2) if not hall else (0, 1, 3)):
        stages = 3 if not hall else 5
        floor = 0.0
        if hall and i:
            floor = rounding_floor(c, "register" if i == 1 else "curl", mb, mu, stages)
        ok, e = field_ok(ctx.get_vec(dev[i]), host[i], 1e-12, floor)
        assert ok, (i, e)
    ctx.close()
