"""Device memory of an adjoint sweep: it takes no more than the checkpoints, the stage states of a
segment and sixteen further fields of the records' size beside the fused state -- what it took when
it worked on the caller's records -- so that a sweep that fits the device goes on fitting."""
from __future__ import annotations

import math

import numpy as np
import pytest

from tests.helpers import maps_for

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def _used(c, steps, every):
    import torch
    ctx = maps_for(c).context()
    b, u, lam = ctx.vec(), ctx.vec(), ctx.vec()
    ctx.kernel("init_b", b)
    ctx.kernel("init_u", u)
    ctx.kernel("init_b", lam)
    rho = ctx.scalar(np.ones(ctx.n_pad))
    ctx.synchronize()
    before = torch.cuda.mem_get_info()[0]
    ctx.adjoint_steps(b, lam, u, rho, steps, every)
    ctx.synchronize()
    used = before - torch.cuda.mem_get_info()[0]
    n = ctx.n_pad
    ctx.close()
    return used, n


@pytest.mark.parametrize("kernel", ["AUTO", "LIST"])
@pytest.mark.parametrize("integrator, stages", [("SSPRK33", 3), ("CarpenterKennedy2N54", 5)])
@pytest.mark.parametrize("variable_u", [False, True])
def test_memory_of_a_sweep(integrator, stages, variable_u, kernel):
    c = dict(order=4, testcase="hall_periodic", nodes=(64, 64, 64), lo=0.0, hi=4 * math.pi / 3, periodic=True, hall=True,
             integrator=integrator, dt=1e-3, variable_u=variable_u, stage_kernel=kernel)
    _used(dict(c, nodes=(16, 16, 16)), 4, 2)   # what the process loads once
    used, n = _used(c, 8, 4)
    fields = 2 + stages * 4 + 16
    # every field a whole number of 2 MiB pages; the state's 27 planes; a page for what is smaller
    assert used <= fields * 32 * n + 27 * 8 * n + 4 * MIB
