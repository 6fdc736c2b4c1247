"""A grid barrier of the CG loop whose wait runs out (it is told to wait for one block more than the
grid has, with a short limit): the cleaning reports IEQ_ERR_TIMEOUT and leaves the field as it
was, and the next cleaning of the context gives what one without a time-out gives."""
from __future__ import annotations

import numpy as np
import pytest

from inductioneq_b200.lib import IeqError
from tests.helpers import maps_for, rel_err

pytestmark = pytest.mark.gpu

CASE = dict(order=4, testcase="confined_domain", nodes=(37, 22, 20), lo=0.0, hi=1.0, hall=True,
            integrator="CarpenterKennedy2N54", dt=1e-5, laplace="WIDE_STENCIL_DIRICHLET")
SPINS = 2000


def _field(ctx):
    b = ctx.vec()
    ctx.kernel("init_b", b)
    bh = ctx.get_vec(b)
    bh[: ctx.n, :3] += 1e-2 * np.random.default_rng(7).random((ctx.n, 3))
    return bh


def test_cleaning_whose_barrier_gives_up_leaves_the_field():
    ctx, ref = maps_for(CASE).context(), maps_for(CASE).context()
    bh = _field(ctx)
    b = ctx.vec(bh)
    ctx.test_cg_barrier(1, SPINS)
    for _ in range(2):
        with pytest.raises(IeqError) as e:
            ctx.clean_div(b, 10, 1e-14, check=False)
        assert e.value.name == "IEQ_ERR_TIMEOUT"
        np.testing.assert_array_equal(ctx.get_vec(b), bh)
    ctx.test_cg_barrier(0)
    res = ctx.clean_div(b, 10, 1e-14, check=False)
    rb = ref.vec(bh)
    want = ref.clean_div(rb, 10, 1e-14, check=False)
    assert res == want and res["iterations"] == 10
    np.testing.assert_array_equal(ctx.get_vec(b), ref.get_vec(rb))
    assert np.abs(ctx.get_vec(b) - bh).max() > 1e-6
    ctx.close()
    ref.close()


def test_time_loop_whose_cleanings_give_up_steps_without_them():
    out = []
    for cleaned in (True, False):
        ctx = maps_for(CASE).context()
        f = [ctx.vec(_field(ctx)), ctx.vec(), ctx.vec(), ctx.vec(), ctx.vec(), ctx.scalar(np.ones(ctx.n_pad)),
             ctx.scalar(np.zeros(2), n=2)]
        if cleaned:
            ctx.test_cg_barrier(1, SPINS)
            with pytest.raises(IeqError) as e:
                ctx.time_steps_integrals(*f, 3, 5, 1e-14)
            assert e.value.name == "IEQ_ERR_TIMEOUT"
        else:
            ctx.time_steps(*f, 3)
        out.append(ctx.get_vec(f[0]))
        if cleaned:   # and the context cleans again
            ctx.test_cg_barrier(0)
            res = ctx.clean_div(f[0], 5, 1e-14, check=False)
            assert res["iterations"] == 5
            assert np.abs(ctx.get_vec(f[0]) - out[0]).max() > 1e-6
        ctx.close()
    assert rel_err(out[0], out[1]) <= 1e-13   # (the loop's first curl kernel also forms the diagnostics)
