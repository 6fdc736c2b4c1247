"""The one-launch CG loop (cg.cuh) against the oracle's host loop (clean_div.m) where its tiles
can go wrong: grids smaller than a tile, tiles and chunks with remainders in every axis, the
narrowest and the widest Laplacians (one and two rows per thread), periodic wraps, a grid whose
tiles outnumber the resident blocks, a field that is clean already and a cap of zero.

Tolerances are those of the cleaning's other parity tests: the same iteration count, the field
to 1e-11 of its scale, the residual to 1e-6 (its value after k iterations carries the rounding
of every dot product before it)."""
from __future__ import annotations

import numpy as np
import pytest

from oracle.hostloops import clean_div
from tests.golden.cases import NOISE_SEED
from tests.helpers import maps_for, oracle_for, rel_err

pytestmark = pytest.mark.gpu

WSD, NSD, LNS = "WIDE_STENCIL_DIRICHLET", "NARROW_STENCIL_DIRICHLET", "WIDE_STENCIL_LNS"
# nodes, order, extended, laplace, periodic, iterations
CASES = [((5, 6, 7), 2, False, NSD, False, 6),        # W = 3, less than a tile
         ((35, 18, 9), 2, False, WSD, False, 8),      # W = 5, one column and one row over
         ((34, 19, 12), 4, False, NSD, False, 8),     # W = 5
         ((33, 35, 13), 2, True, LNS, False, 8),      # W = 7, no Dirichlet layer
         ((67, 34, 21), 4, False, WSD, False, 10),    # W = 9, three x tiles
         ((36, 20, 24), 6, False, NSD, False, 8),     # W = 9
         ((40, 17, 15), 4, False, LNS, False, 8),     # W = 11
         ((37, 23, 19), 4, True, WSD, False, 8),      # W = 13
         ((30, 29, 31), 6, False, WSD, False, 8),     # W = 15
         ((34, 18, 20), 6, False, LNS, False, 6),     # W = 17
         ((41, 18, 17), 6, True, WSD, False, 6),      # W = 19
         ((20, 33, 18), 6, True, LNS, False, 6),      # W = 21
         ((9, 34, 11), 4, False, WSD, True, 8),       # periodic wraps
         ((38, 21, 17), 6, False, WSD, True, 6),
         ((300, 260, 13), 6, False, WSD, False, 2)]   # 330 tiles: more than one a block


def _run(c, iters, thr=1e-13, noise=0.01):
    o = oracle_for(c)
    b = o.vec()
    o.run("init_b", o.cfg.nodes, b)
    b[:, :3] += noise * np.random.default_rng(NOISE_SEED).random((o.N, 3))
    ctx = maps_for(c).context()
    db = ctx.vec(b)
    ref = b.copy()
    r = clean_div(o, ref, iters, thr, c["bnodes"])
    res = ctx.clean_div(db, iters, thr, check=False)
    got = ctx.get_vec(db)[: o.N]
    ctx.close()
    return r, res, got, ref


@pytest.mark.parametrize("nodes, order, extended, laplace, periodic, iters", CASES)
def test_cg_loop_matches_host_loop(nodes, order, extended, laplace, periodic, iters):
    c = dict(order=order, extended=extended, testcase="confined_domain", nodes=nodes, lo=0.0, hi=1.0,
             laplace=laplace, bnodes=0 if laplace == LNS else 1, periodic=periodic)
    r, res, got, ref = _run(c, iters)
    assert res["iterations"] == r["iterations"]
    assert abs(res["residual_norm2"] - r["residual_norm2"]) <= 1e-6 * r["residual_norm2"]
    assert abs(res["divergence_norm_initial"] - r["initial_norm"]) <= 1e-12 * r["initial_norm"]
    assert rel_err(got, ref) <= 1e-11


def test_cg_loop_stops_before_the_first_iteration():
    c = dict(order=4, testcase="confined_domain", nodes=(20, 18, 22), lo=0.0, hi=1.0, laplace=WSD, bnodes=1)
    for iters, thr in ((0, 1e-13), (5, 1e6)):
        r, res, got, ref = _run(c, iters, thr)
        assert res["iterations"] == r["iterations"] == 0
        assert rel_err(got, ref) <= 1e-15
