"""The operator constants compiled into the box kernels (struct Op in ieq_common.cuh) against the
operators' rows: the list lengths ND and NU, the reach QX in pairs along x, and no derivative
coefficient outside a box; and that the library accepts every operator."""
from __future__ import annotations

import copy
import ctypes
import json
import os
import re

import pytest

from inductioneq_b200 import lib as L

PKG = os.path.dirname(os.path.abspath(L.__file__))
OPS = ["2c", "4c", "6c", "2e", "4e", "6e"]


def _constants():
    out = {}
    with open(os.path.join(PKG, "csrc", "ieq_common.cuh")) as f:
        for m in re.finditer(r"struct Op<(\d)> \{ static constexpr int ([^;]*);", f.read()):
            out[OPS[int(m.group(1))]] = {k.strip(): int(v) for k, v in (p.split("=") for p in m.group(2).split(","))}
    assert sorted(out) == sorted(OPS)
    return out


def _rows(t):
    """The 2 nb + 1 rows of a table: left boundary rows, the interior row and the mirrored right
    ones, as {offset: coefficient} of the non-zero entries."""
    nb, c0 = t["nb"], (t["width"] - 1) // 2
    left = [{k - c0: v for k, v in enumerate(map(float.fromhex, r)) if v != 0.0} for r in t["rows"][: nb + 1]]
    return left + [{-o: t["sign"] * v for o, v in left[2 * nb - r].items()} for r in range(nb + 1, 2 * nb + 1)]


def faults(op, c):
    """What in the operator's rows the constants c do not cover."""
    bad = []
    nb, wh = op["nb"], op["w_hod"]
    if (nb, op["sw"], wh) != (c["NB"], c["SW"], c["WH"]):
        bad.append("sizes")
    D = _rows(op["D"])
    dho = [list(map(float.fromhex, r)) for r in op["DHO"]["rows"]]
    dho += [dho[2 * nb - r][::-1] for r in range(nb + 1, 2 * nb + 1)]
    for r, row in enumerate(D):
        H = {s + i for s in range(-wh + 1, 1) for i in range(wh) if dho[r][s + wh - 1] != 0.0 and dho[nb][i] != 0.0}
        if len(row) > c["ND"]:
            bad.append(f"ND of row {r}")
        if len(set(row) | H) > c["NU"]:
            bad.append(f"NU of row {r}")
        for o in row:
            if (r < nb and r + o < 0) or (r > nb and o > 2 * nb - r):
                bad.append(f"row {r} leaves the box at {o}")
            # even rows: node r is the first or second of its pair, the node d from the end the other way round
            for k in (r % 2,) if r < nb else (0, 1) if r == nb else (1 - (2 * nb - r) % 2,):
                if not -2 * c["QX"] - k <= o <= 2 * c["QX"] + 1 - k:
                    bad.append(f"QX of row {r}")
            # odd rows: one pair further, the nodes at the end paired like those at the start
            if r > nb and not -2 * (c["QX"] + 1) - r % 2 <= o <= 2 * (c["QX"] + 1) + 1 - r % 2:
                bad.append(f"QX of row {r} of odd rows")
    return bad


def _tables():
    with open(os.path.join(PKG, "sbp_tables.json")) as f:
        return json.load(f)


@pytest.mark.parametrize("name", OPS)
def test_constants_cover_the_operator(name):
    assert faults(_tables()[name], _constants()[name]) == []


@pytest.mark.parametrize("name", OPS)
@pytest.mark.parametrize("key", ["ND", "NU", "QX"])
def test_a_smaller_constant_is_found(name, key):
    c = dict(_constants()[name])
    c[key] -= 1
    assert faults(_tables()[name], c) != []


def test_a_coefficient_outside_the_box_is_found():
    t = copy.deepcopy(_tables()["4c"])
    t["D"]["rows"][0][0] = (0.25).hex()
    assert any("leaves the box" in f for f in faults(t, _constants()["4c"]))


@pytest.mark.parametrize("name", OPS)
def test_the_library_takes_every_operator(name):
    # (a grid too short for it: refused for that, after the rows were looked at)
    so = L.load()
    paths = [f"../include/{name[0]}{'nd' if name[0] == '2' else 'th'}Order{'Extended' if name[1] == 'e' else ''}.h",
             "../include/rotation_3D.h"]
    arr = (ctypes.c_char_p * 2)(*[p.encode() for p in paths])
    h = ctypes.c_void_p()
    s = " -DNODES_X=1 -DNODES_Y=1 -DNODES_Z=1 -DXMIN=0 -DXMAX=1 -DYMIN=0 -DYMAX=1 -DZMIN=0 -DZMAX=1"
    assert so.ieq_create(ctypes.byref(h), s.encode(), arr, 2, 0) == 2
    assert "2*NUM_BOUNDS" in so.ieq_last_error(None).decode()
