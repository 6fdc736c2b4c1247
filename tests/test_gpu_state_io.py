"""Entry and exit of the fused calls, which convert only what a step reads and writes: registers
and curl buffers full of NaN on entry do not matter, u may turn zero and back between the calls
of one context (the conversion of u rides on the look at it only if the last call found it
non-zero), graphs of earlier calls are used again, on grids with and without a row pitch; and
the time loop with cleaning on the state in place equals the one on the caller's records."""
from __future__ import annotations

import numpy as np
import pytest

from tests.helpers import maps_for, rel_err

pytestmark = pytest.mark.gpu

INTEGRATORS = ["SSPRK33", "SSPRK104", "KennedyCarpenterLewis2R54C", "CalvoFrancoRandez2R64",
               "CarpenterKennedy2N54", "ToulorgeDesmet2N84F"]


def _case(nodes, integrator, hall):
    return dict(order=4, testcase="confined_domain" if hall else "rotation_3D", nodes=nodes, lo=0.0 if hall else -1.0,
                hi=1.0, hall=hall, integrator=integrator, dt=1e-4)


def _fields(ctx, b, u):
    bad = np.full((ctx.n_pad, 4), np.nan)
    return [ctx.vec(b), ctx.vec(bad), ctx.vec(bad), ctx.vec(bad if ctx_hall(ctx) else None), ctx.vec(u),
            ctx.scalar(np.linspace(0.8, 1.3, ctx.n_pad)), ctx.scalar(np.zeros(2), n=2)]


def ctx_hall(ctx):
    return ctx.hall


@pytest.mark.parametrize("hall", [False, True])
@pytest.mark.parametrize("nodes", [(17, 13, 12), (18, 13, 12)])
@pytest.mark.parametrize("integrator", INTEGRATORS)
def test_calls_that_change_u_equal_fresh_contexts(integrator, nodes, hall):
    c = _case(nodes, integrator, hall)
    ctx = maps_for(c).context()
    ctx.hall = hall
    rng = np.random.default_rng(3)
    b0 = rng.standard_normal((ctx.n_pad, 4))
    b0[:, 3] = 0.0
    u1 = 0.3 * rng.standard_normal((ctx.n_pad, 4))
    u1[:, 3] = 0.0
    one = np.zeros_like(u1)
    one[ctx.n - 1, 2] = 0.25   # a single non-zero value, in the last node
    dev = _fields(ctx, b0, u1)
    b = b0
    for k, u in enumerate((u1, np.zeros_like(u1), one, np.zeros_like(u1), u1)):
        dev[4].upload(u)
        steps = 1 + k % 3
        ctx.time_steps(*dev, steps)
        fresh = maps_for(c).context()
        fresh.hall = hall
        other = _fields(fresh, b, u)
        other[6].upload(np.zeros(2))
        t = ctx.get_scalar(dev[6], n=2)
        fresh.time_steps(*other, steps)
        b = ctx.get_vec(dev[0])
        assert np.isfinite(b).all()
        if k == 0 or hall:   # (the inflow data of a box without the Hall term depends on the time)
            np.testing.assert_array_equal(b, fresh.get_vec(other[0]))
            np.testing.assert_array_equal(ctx.get_vec(dev[1]), fresh.get_vec(other[1]))
            if hall:
                np.testing.assert_array_equal(ctx.get_vec(dev[3])[: ctx.n], fresh.get_vec(other[3])[: ctx.n])
        assert t[0] > 0
        fresh.close()
    ctx.close()


@pytest.mark.parametrize("nodes", [(21, 18, 19), (22, 18, 19)])
def test_cleaned_series_in_place_equals_records(nodes):
    out = []
    for form in (2, 1):
        c = dict(_case(nodes, "CarpenterKennedy2N54", True), laplace="WIDE_STENCIL_DIRICHLET", cg_pass_a=form,
                 dissipation="HIGH_ORDER", dt=2e-5)
        ctx = maps_for(c).context()
        ctx.hall = True
        b = ctx.vec()
        ctx.kernel("init_b", b)
        bh = ctx.get_vec(b)
        bh[: ctx.n, :3] += 0.01 * np.random.default_rng(7).random((ctx.n, 3))
        dev = _fields(ctx, bh, np.zeros_like(bh))
        ctx.kernel("init_u", dev[4])
        res = ctx.time_steps_integrals(*dev, 3, 12, 1e-12)
        out.append((res, ctx.get_vec(dev[0]), ctx.get_vec(dev[3])[: ctx.n]))
        ctx.close()
    for k in ("energy", "divergence_norm", "l2_error"):
        np.testing.assert_allclose(out[0][0][k], out[1][0][k], rtol=1e-9)
    assert rel_err(out[0][1], out[1][1]) <= 1e-11
    assert rel_err(out[0][2], out[1][2]) <= 1e-9   # (a derivative of the field above: 1 / dx larger)
