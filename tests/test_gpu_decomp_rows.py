"""The z-slab decomposition against the undecomposed run, bit for bit, where the two run different
kernels: boxes with odd rows (the undecomposed state has a row pitch and takes the node-pair
kernels, with the x boundary columns in a launch of their own where they pay; a slab's state has
none and takes the one-node kernels), and adaptive dissipation, whose block shape depends on the
size of the grid and whose warps hold other nodes then."""
from __future__ import annotations

import math

import numpy as np
import pytest

from inductioneq_b200 import ranks as R
from inductioneq_b200.decomp import SlabSolve, run_local
from tests.helpers import maps_for

pytestmark = pytest.mark.gpu

SP, CE, ZE, PR = "SPLIT", "CENTRAL", "ZERO", "PRODUCT"
STEPS = 2


def _rotation(nodes, order, **kw):
    return dict(order=order, testcase="rotation_3D", nodes=nodes, lo=-1.0, hi=1.0, integrator="SSPRK33", dt=3e-3, **kw)


def _hall(nodes, order, **kw):
    return dict(order=order, testcase="hall_periodic", nodes=nodes, lo=0.0, hi=1.0, hall=True,
                integrator="CarpenterKennedy2N54", dt=1e-5, **kw)


def _confined(nodes, order, **kw):
    return dict(order=order, testcase="confined_domain", nodes=nodes, lo=0.0, hi=1.0, hall=True,
                integrator="CarpenterKennedy2N54", dt=1e-3, **kw)


def _start(c, noise, share):
    """(b, u) on the host: the testcase's fields with noise on a share of the nodes."""
    g = maps_for(c).context()
    b, u = g.vec(), g.vec()
    g.kernel("init_b", b)
    g.kernel("init_u", u)
    bh, uh = g.get_vec(b), g.get_vec(u)
    rng = np.random.default_rng(3)
    bh[: g.n, :3] += noise * rng.standard_normal((g.n, 3)) * (rng.random((g.n, 1)) < share)
    n = g.n
    g.close()
    return bh[:n], uh[:n]


def _whole(c, bh, uh):
    g = maps_for(c).context()
    dev = [g.vec(), g.vec(), g.vec(), g.vec(), g.vec(), g.scalar(np.ones(g.n_pad)), g.scalar(np.zeros(2), n=2)]
    dev[0].upload(bh)
    dev[4].upload(uh)
    g.time_steps(*dev, STEPS)
    out = [g.get_vec(dev[k])[: g.n] for k in range(3)]
    g.close()
    return out


def _compare(c, world, noise=1e-2, share=1.0):
    bh, uh = _start(c, noise, share)
    ref = _whole(c, bh, uh)
    assert np.abs(ref[0] - bh).max() > 0
    solves = [SlabSolve(maps_for(c), R.Ranks(world, r, r)) for r in range(world)]
    try:
        for s in solves:
            s.load(bh, uh, np.ones(bh.shape[0]))
        run_local(solves, STEPS) if world > 1 else solves[0].steps(STEPS)
        for s in solves:
            rows = s.slabs.global_rows()
            for got, want in zip((s.b, s.b2, s.b3)[: s.nf], ref):
                np.testing.assert_array_equal(s.owned(got), want[rows])
    finally:
        for s in solves:
            s.close()


ODD = [_rotation((nx, 14, 36), o) for o in (2, 4, 6) for nx in (41, 97)]
# every flux-form mask that has a pair kernel, and one that has none
ODD += [_rotation((33, 15, 36), 4, uibj=a, source=b, ujbi=c)
        for a, b, c in ((PR, CE, CE), (CE, ZE, PR), (SP, CE, SP), (SP, ZE, CE), (CE, CE, SP), (SP, ZE, PR), (CE, ZE, CE))]
ODD += [_rotation((41, 14, 36), o, dissipation=d) for o in (4, 6) for d in ("FIRST_ORDER", "HIGH_ORDER")]
ODD += [_confined((nx, 14, 36), o, dissipation=d) for o in (2, 4, 6) for nx in (41, 97) for d in ("NONE", "HIGH_ORDER")]
ODD += [_hall((41, 14, 36), o, dissipation=d) for o in (4, 6) for d in ("NONE", "FIRST_ORDER", "HIGH_ORDER")]
ODD += [_rotation((41, 14, 36), o, real="float") for o in (2, 6)] + [_confined((41, 14, 36), 4, real="float")]
ODD += [dict(_rotation((41, 14, 36), 4), testcase=t, hall=False) for t in ("rotation_2D", "rotation_gaussian")]


@pytest.mark.parametrize("world", [1, 3])
@pytest.mark.parametrize("c", ODD)
def test_slabs_of_odd_rows_equal_the_whole_grid(c, world):
    _compare(c, world)


@pytest.mark.parametrize("order", [2, 4, 6])
@pytest.mark.parametrize("make", [_rotation, _hall])
def test_slabs_with_adaptive_dissipation_equal_the_whole_grid(make, order):
    # 64 x 64 x 72: above the size from which the blocks are compact, its slabs of two below it;
    # steep places in a five-hundredth of the nodes, so that warps hold quiet and loud nodes
    _compare(make((64, 64, 72), order, dissipation="ADAPTIVE"), 2, noise=0.5, share=0.002)


@pytest.mark.parametrize("real", ["double", "float"])
@pytest.mark.parametrize("order, extended", [(2, False), (4, False), (6, False), (4, True)])
@pytest.mark.parametrize("periodic", [False, True])
def test_adaptive_dissipation_does_not_depend_on_the_block_shape(order, extended, periodic, real):
    c = dict(_hall((37, 18, 20), order, dissipation="ADAPTIVE", real=real, extended=extended, periodic=periodic),
             hi=4 * math.pi / 3, dt=1e-4)
    bh, uh = _start(c, 0.5, 0.01)
    ref = _whole(dict(c, col_block=(32, 4, 1)), bh, uh)
    for shape in ((8, 8, 2), (128, 1, 1), (1, 128, 1)):
        for got, want in zip(_whole(dict(c, col_block=shape), bh, uh), ref):
            np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("nodes", [(40, 14, 20), (97, 14, 20)])
@pytest.mark.parametrize("order", [2, 4, 6])
@pytest.mark.parametrize("make, kw", [(_rotation, {}), (_rotation, dict(uibj=SP, source=CE, ujbi=SP)),
                                      (_rotation, dict(dissipation="FIRST_ORDER")), (_confined, {}),
                                      (_hall, dict(dissipation="HIGH_ORDER"))])
def test_stage_kernels_of_one_and_two_nodes_and_bands_round_alike(make, kw, order, nodes):
    c = make(nodes, order, **kw)
    if make is _confined:
        c["dt"] = 1e-5
    bh, uh = _start(c, 1e-2, 1.0)
    ref = _whole(c, bh, uh)
    for other in (dict(col_pairs=0), dict(xband=0), dict(xband=2)):
        for got, want in zip(_whole(dict(c, **other), bh, uh), ref):
            np.testing.assert_array_equal(got, want)
