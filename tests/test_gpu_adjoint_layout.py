"""The checkpointed adjoint on the planes of the fused state: odd rows (padded planes), the
wall-free periodic kernels and the general ones, SSPRK33 running from kept stage state to kept
stage state and the schemes that copy them, against the same sweep on the reference kernel
lists, which works on the caller's records.

Both linearise about the same trajectory up to rounding, in other orders of summation: a few
hundred operations of relative 1.1e-16 a stage, some 60 stages, so the gradients agree to 1e-11
of their scale.
"""
from __future__ import annotations

import math

import numpy as np
import pytest

from tests.helpers import maps_for

pytestmark = pytest.mark.gpu

HP = 4.0 * math.pi / 3.0
WAVE = dict(testcase="hall_periodic", lo=0.0, hi=HP, periodic=True, hall=True, integrator="SSPRK33")
BOX = dict(testcase="rotation_gaussian", lo=-1.0, hi=1.0, integrator="SSPRK33")
CASES = {
    "plain_2_odd": dict(WAVE, order=2, nodes=(17, 16, 19), variable_u=True),
    "plain_4_odd": dict(WAVE, order=4, nodes=(33, 17, 18), variable_u=True),
    "plain_4_fixed_u": dict(WAVE, order=4, nodes=(35, 16, 17)),
    "plain_6": dict(WAVE, order=6, nodes=(18, 17, 16), variable_u=True),
    "periodic_hod_odd": dict(WAVE, order=4, nodes=(17, 18, 16), dissipation="HIGH_ORDER"),
    "periodic_split_odd": dict(WAVE, order=4, nodes=(19, 18, 16), uibj="SPLIT", source="SPLIT", ujbi="SPLIT"),
    "periodic_2n_odd": dict(WAVE, order=4, nodes=(17, 16, 18), integrator="CarpenterKennedy2N54", variable_u=True),
    "box_odd": dict(BOX, order=6, nodes=(35, 14, 15)),
    "box_hall_odd": dict(order=4, testcase="hall_travelling_wave", nodes=(15, 14, 16), lo=0.0, hi=2 * math.pi,
                         hall=True, integrator="SSPRK33"),
    "box_fo_odd": dict(BOX, order=2, nodes=(13, 12, 11), dissipation="FIRST_ORDER"),
    # u = 0 and a grid the tiled brick kernels take: their tensor maps name the state's own
    # buffers, so SSPRK33's stage states are copied out
    "brick": dict(order=4, testcase="hall_circular_wave", nodes=(32, 32, 32), lo=-1.0, hi=1.0, periodic=True, hall=True,
                  integrator="SSPRK33", dissipation="HIGH_ORDER", kernel="BRICK"),
}


def _gradient(c, dt, kernel, steps, every, passes=1):
    ctx = maps_for(dict(c, dt=dt, stage_kernel=kernel)).context()
    b, u = ctx.vec(), ctx.vec()
    ctx.kernel("init_b", b)
    ctx.kernel("init_u", u)
    lam0 = np.zeros((ctx.n_pad, 4))
    lam0[: ctx.n, :3] = np.random.default_rng(5).standard_normal((ctx.n, 3))
    rho = np.ones(ctx.n_pad)
    rho[: ctx.n] += 0.1 * np.random.default_rng(6).random(ctx.n)
    for _ in range(passes):
        lam = ctx.vec(lam0)
        ctx.adjoint_steps(b, lam, u, ctx.scalar(rho), steps, every)
    out = ctx.get_vec(lam)[: ctx.n, :3].copy()
    ctx.close()
    return out


@pytest.mark.parametrize("name", sorted(CASES))
def test_sweep_on_planes_equals_sweep_on_records(name):
    c = dict(CASES[name])
    kernel = c.pop("kernel", "AUTO")
    dt = 0.05 * (c["hi"] - c["lo"]) / max(c["nodes"])
    # 7 steps with checkpoints every 3: a last segment of one step
    ref = _gradient(c, dt, "LIST", 7, 3)
    got = _gradient(c, dt, kernel, 7, 3, passes=2)
    assert np.isfinite(ref).all() and np.abs(ref).max() > 0
    assert np.abs(got - ref).max() <= 1e-11 * np.abs(ref).max()
