"""Grids beyond what 32 bits of node index or 65,535 blocks of a launch reach: the kernels on the
caller's records (operators, kernel lists, results, cleaning) on fields of more than 2^31 nodes,
and grids with a very long axis, whose block shapes must stay within a launch's limits.  A part of
a large field is compared with the same kernel on a small grid that is that part."""
from __future__ import annotations

import numpy as np
import pytest

from tests.helpers import maps_for, rel_err

pytestmark = pytest.mark.gpu

N = 1300                # N^3 = 2.197e9 nodes; the last 29 planes lie beyond 2^31
PART = 24               # planes of the part, of which the middle ones are compared
LOW = slice(6, 18)


def _setup(fields):
    """Two FP32 periodic contexts with spacing 1, the large grid's and the part's, or a skip where
    the device has no room for `fields` records and the cleaning's vectors."""
    import torch
    n = N ** 3
    if torch.cuda.mem_get_info()[0] < n * fields * 16 + (4 << 30):
        pytest.skip("the device has no room for the fields")
    c = dict(order=4, testcase="hall_periodic", nodes=(N, N, N), lo=0.0, hi=float(N), periodic=True, real="float",
             integrator="CarpenterKennedy2N54", dt=0.125, laplace="WIDE_STENCIL_DIRICHLET")
    m = maps_for(c)
    big = m.context()
    p = maps_for(c)
    p.I_Mesh.update({"NODES_Z": PART, "ZMAX": float(PART)})
    return big, p.context()


def _rand(seed, rows):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    t = torch.empty((rows, 4), dtype=torch.float32, device="cuda")
    for k in range(0, rows, 1 << 26):   # (in pieces: torch's own generators index a call in 32 bits)
        t[k:k + (1 << 26)].uniform_(-1.0, 1.0, generator=g)
    t[:, 3] = 0
    return t


def _planes(t, z0, planes, plane):
    return t[z0 * plane:(z0 + planes) * plane]


@pytest.mark.parametrize("kernel", ["calc_curl", "CarpenterKennedy2N54_1a"])
def test_kernels_on_records_of_more_than_2_31_nodes(kernel):
    import torch
    stage = kernel != "calc_curl"
    big, part = _setup(3 if stage else 2)
    plane, n = N * N, N ** 3
    b = _rand(1, n)
    u = _rand(2, n) if stage else None
    out = torch.zeros((n, 4), dtype=torch.float32, device="cuda")
    small = torch.zeros((PART * plane, 4), dtype=torch.float32, device="cuda")
    time = torch.zeros(2, dtype=torch.float32, device="cuda")
    z0 = N - PART
    assert (z0 + LOW.start) * plane > 2 ** 31
    torch.cuda.synchronize()
    if stage:   # (without the Hall term the list reads neither the curl buffer nor rho)
        big.kernel(kernel, b, out, out, u, time, time)
        part.kernel(kernel, _planes(b, z0, PART, plane), small, small, _planes(u, z0, PART, plane), time, time)
    else:
        big.kernel(kernel, b, out)
        part.kernel(kernel, _planes(b, z0, PART, plane), small)
    big.synchronize()
    part.synchronize()
    rows = slice(LOW.start * plane, LOW.stop * plane)
    got, want = _planes(out, z0, PART, plane)[rows], small[rows]
    assert bool((want[:, :3].abs().amax(0) > 0).all())
    # the same operations on the same values
    assert torch.equal(got, want)
    big.close()
    part.close()
    del b, u, out, small, got, want
    torch.cuda.empty_cache()


def test_results_of_more_than_2_31_nodes():
    import torch
    big, part = _setup(4)
    n = N ** 3
    b = _rand(3, n)
    wv = torch.empty((n, 4), dtype=torch.float32, device="cuda")
    ws, div = (torch.empty(n, dtype=torch.float32, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    res = big.results(b, 0.0, wv, ws)
    big.kernel("calc_div", b, div)
    big.synchronize()
    # (a sum of 2.2e9 FP32 terms in FP64, in two orders)
    assert abs(res["energy"] - big.norm2(b)) <= 1e-9 * res["energy"]
    assert abs(res["divergence_norm"] - big.norm2_S(ws) ** 0.5) <= 1e-9 * res["divergence_norm"]
    assert abs(res["abs_err"] - big.norm2_diff(b, wv) ** 0.5) <= 1e-9 * res["abs_err"]
    tail = slice(2 ** 31 + 1, n)
    d, w = div[tail], ws[tail]
    # div B of the results against calc_div: sums of up to 12 terms in FP32
    assert float((d - w).abs().max()) <= 12 * 2.0 ** -23 * float(d.abs().max())
    assert float(d.abs().max()) > 0.1
    big.close()
    part.close()
    del b, wv, ws, div, d, w
    torch.cuda.empty_cache()


def test_cleaning_of_more_than_2_31_nodes():
    # one CG iteration adds alpha grad(div B): alpha is one number for the whole grid, so the
    # change of a part is the part's own change times the ratio of the two alphas
    import torch
    big, part = _setup(4.1)
    plane, n = N * N, N ** 3
    b = _rand(4, n)
    z0 = N - PART
    before = _planes(b, z0, PART, plane).clone()
    small = before.clone()
    torch.cuda.synchronize()
    res = big.clean_div(b, 1, 1e-30, check=False)
    part.clean_div(small, 1, 1e-30, check=False)
    assert res["iterations"] == 1
    rows = slice(LOW.start * plane, LOW.stop * plane)
    got = (_planes(b, z0, PART, plane) - before)[rows, :3].double()
    want = (small - before)[rows, :3].double()
    ratio = float((got * want).sum() / (want * want).sum())
    scale = float(got.abs().max())
    assert scale > 1e-2
    # B of order 1 in FP32, rounded once on each side
    assert float((got - ratio * want).abs().max()) <= 2.0 ** -23 * (1 + abs(ratio)) * (1 + scale)
    big.close()
    part.close()
    del b, before, small, got, want
    torch.cuda.empty_cache()


def _long(order, nodes, integrator="CarpenterKennedy2N54", **kw):
    return dict(order=order, testcase=kw.pop("testcase", "rotation_3D"), nodes=nodes, lo=-1.0, hi=1.0,
                integrator=integrator, dt=1e-7, **kw)


def _advance(c, steps=1):
    ctx = maps_for(c).context()
    rng = np.random.default_rng(6)
    b, u = (ctx.vec(rng.standard_normal((ctx.n_pad, 4)) * [1, 1, 1, 0]) for _ in range(2))
    f = [b, ctx.vec(), ctx.vec(), ctx.vec(), u, ctx.scalar(np.ones(ctx.n_pad)), ctx.scalar(np.zeros(2), n=2)]
    ctx.time_steps(*f, steps)
    out = ctx.get_vec(f[0])
    ctx.close()
    return out


@pytest.mark.parametrize("case, other", [
    # the kernel lists against the fused kernels (the list's other kernels end at 262,140 rows)
    (_long(2, (4, 200000, 4), stage_kernel="LIST"), {"stage_kernel": "AUTO"}),
    # the default block shapes against one given
    (_long(2, (4, 600000, 4), dissipation="ADAPTIVE"), {"col_block": (4, 32, 1)}),
    (_long(2, (4, 600000, 4), dissipation="HIGH_ORDER"), {"col_block": (4, 32, 1)})])
def test_very_long_axes(case, other):
    assert rel_err(_advance(case), _advance(dict(case, **other))) <= 1e-13


def test_adjoint_of_a_very_long_axis():
    # <F'^T w, v> = <w, F' v>
    c = _long(2, (4, 200000, 4), testcase="confined_domain", hall=True)
    ctx = maps_for(c).context()
    rng = np.random.default_rng(5)
    b, v, w, u = (ctx.vec(rng.standard_normal((ctx.n_pad, 4))) for _ in range(4))
    rho = ctx.scalar(np.ones(ctx.n_pad))
    jv, jtw = ctx.vec(), ctx.vec()
    ctx.operator_jvp(b, v, u, rho, jv)
    ctx.operator_vjp(b, w, u, rho, jtw)
    hv, hw, hjv, hjtw = (ctx.get_vec(x)[: ctx.n, :3] for x in (v, w, jv, jtw))
    left, right = float((hjtw * hv).sum()), float((hw * hjv).sum())
    assert abs(left - right) <= 1e-11 * float(np.abs(hw * hjv).sum())
    ctx.close()
