"""The workloads that this framework is timed on, through its public entry points.

A case is a dict of plain values.  Its ``kind`` says which entry point it goes through:

  steps    ``Context.time_steps``: the fused time loop of one solve
  series   ``Context.time_steps_integrals``: the time loop with the diagnostics of every step
           and the divergence cleaning after it
  clean    ``Context.clean_div``: the projection of one field
  list     ``Context.run`` with one step's reference kernel list, and ``Context.results``
  adjoint  ``Context.adjoint_steps``: the gradient through a checkpointed run
  batch    ``Batch.run``: many independent solves of uneven sizes

``prepare`` makes what a program holds before the call (a context, its fields on the GPU),
``run`` makes the call, ``exact`` computes the same outputs in 64 bits with dense derivative
matrices and plain torch operations (the adjoint by automatic differentiation of that).
"""
from __future__ import annotations

import json
import math
import os

import numpy as np
import torch

from inductioneq_b200.batch import Batch, rotation_batch
from inductioneq_b200.induction_eq import Maps

TWO_PI = 2.0 * math.pi
HALL_PERIOD = 4.0 * math.pi / 3.0   # the period of the hall_periodic testcase

# the flux forms (u_i B_j, source, u_j B_i) of the time loop's volume terms
FORMS = {"default": ("PRODUCT", "CENTRAL", "CENTRAL"), "central": ("CENTRAL", "ZERO", "CENTRAL"),
         "split": ("SPLIT", "SPLIT", "SPLIT"), "product": ("PRODUCT", "CENTRAL", "PRODUCT")}

# testcase -> lower and upper end of the domain, periodic, Hall term, updated velocity
DOMAINS = {"rotation_3D": (-1.0, 1.0, False, False, False),
           "hall_circular_wave": (0.0, TWO_PI, True, True, False),
           "hall_periodic": (0.0, HALL_PERIOD, True, True, True),
           "confined_domain": (0.0, 1.0, False, True, False)}


def _case(kind, testcase, n, order=4, integrator="SSPRK33", steps=1, **more):
    c = {"kind": kind, "testcase": testcase, "nx": n[0], "ny": n[1], "nz": n[2], "order": order, "extended": False,
         "forms": "default", "dissipation": "NONE", "real": "double", "integrator": integrator, "steps": steps}
    c.update(more)
    return c


CK = "CarpenterKennedy2N54"


def listed():
    named = {
        # one step of a small solve: a host that looks at the field after every step
        "step_box_24": _case("steps", "rotation_3D", (24, 24, 24), 4, steps=1),
        # a whole small solve, the testcase to t = 1 as the reference's examples run it
        "solve_box_40": _case("steps", "rotation_3D", (40, 40, 40), 4, steps=60),
        # a point of the convergence sweep over the flux forms: odd rows, 6th order
        "sweep_box_97": _case("steps", "rotation_3D", (97, 97, 97), 6, steps=10, forms="central"),
        # the headline workload: a Hall wave, 6th order with high-order dissipation
        "hall_wave_64": _case("steps", "hall_circular_wave", (64, 64, 64), 6, CK, 20, dissipation="HIGH_ORDER"),
        # the same with fields that do not fit the L2 cache: a production-size solve
        "hall_wave_256": _case("steps", "hall_circular_wave", (256, 256, 256), 6, CK, 4, dissipation="HIGH_ORDER"),
        # the 32-bit state
        "hall_wave_128_f32": _case("steps", "hall_circular_wave", (128, 128, 128), 6, CK, 10,
                                   dissipation="HIGH_ORDER", real="float"),
        # adaptive dissipation with an updated velocity, on a field with a thin current sheet
        "adaptive_64": _case("steps", "hall_periodic", (64, 64, 64), 4, CK, 4, dissipation="ADAPTIVE"),
        # a confined Hall run as the cleaning study runs it: diagnostics and a capped cleaning
        # every step, ragged grid
        "cleaned_series_96": _case("series", "confined_domain", (96, 81, 70), 4, CK, 3, dissipation="HIGH_ORDER",
                                   laplace="WIDE_STENCIL_DIRICHLET", max_iterations=50),
        # one projection of a large field, the wide-stencil Laplacian
        "clean_128": _case("clean", "confined_domain", (128, 128, 128), 4, laplace="WIDE_STENCIL_DIRICHLET",
                           max_iterations=50),
        # a host that drives the reference's kernel names one list per step, and its results
        "kernel_list_48": _case("list", "confined_domain", (48, 48, 48), 4, CK, 2, dissipation="HIGH_ORDER"),
        # the gradient with respect to the initial field
        "adjoint_64": _case("adjoint", "hall_periodic", (64, 64, 64), 4, steps=20, checkpoint=10),
        # a parameter study: independent solves of uneven sizes and orders together
        "batch_12": {"kind": "batch", "solves": 12, "draw": 7, "nmin": 16, "nmax": 96, "steps": 20},
    }
    return [dict(c, name=k) for k, c in named.items()]


def draw(rng):
    def size(lo, hi, ragged=True):
        n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        return tuple(max(lo, min(hi, round(n * (rng.uniform(0.85, 1.18) if ragged else 1.0)))) for _ in range(3))

    def count(n, stages, most=4e7, cap=60):
        return max(1, min(cap, int(most / (n[0] * n[1] * n[2] * stages)) or 1, rng.randint(1, cap)))

    kind = rng.choice(["box", "box", "wave", "wave", "periodic", "confined", "series", "clean", "list", "adjoint",
                       "batch"])
    order = rng.choice([2, 4, 6])
    if kind == "box":
        n = size(17, 160, rng.random() < 0.5)
        return _case("steps", "rotation_3D", n, order, steps=count(n, 3), forms=rng.choice(sorted(FORMS)),
                     extended=rng.random() < 0.25)
    if kind == "wave":
        n = size(32, 240, rng.random() < 0.5)
        return _case("steps", "hall_circular_wave", n, order, CK, count(n, 5, cap=20),
                     dissipation=rng.choice(["HIGH_ORDER", "HIGH_ORDER", "NONE"]), real=rng.choice(["double", "float"]))
    if kind == "periodic":
        n = size(24, 96)
        return _case("steps", "hall_periodic", n, order, CK, count(n, 5, 1e7, 8),
                     dissipation=rng.choice(["ADAPTIVE", "FIRST_ORDER", "HIGH_ORDER"]))
    if kind == "confined":
        n = size(24, 128)
        return _case("steps", "confined_domain", n, order, CK, count(n, 5, 2e7, 10),
                     dissipation=rng.choice(["HIGH_ORDER", "NONE"]), forms=rng.choice(sorted(FORMS)),
                     real=rng.choice(["double", "double", "float"]))
    laplace = rng.choice(["WIDE_STENCIL_DIRICHLET", "WIDE_STENCIL_DIRICHLET", "NARROW_STENCIL_DIRICHLET"])
    if kind == "series":
        n = size(24, 100)
        return _case("series", "confined_domain", n, order, CK, rng.randint(1, 3), dissipation="HIGH_ORDER",
                     laplace=laplace, max_iterations=rng.randint(10, 50))
    if kind == "clean":
        return _case("clean", "confined_domain", size(24, 160), order, laplace=laplace,
                     max_iterations=rng.randint(10, 60))
    if kind == "list":
        return _case("list", rng.choice(["confined_domain", "rotation_3D"]), size(17, 80), order,
                     rng.choice([CK, "SSPRK33"]), rng.randint(1, 3),
                     dissipation=rng.choice(["HIGH_ORDER", "NONE"]))
    if kind == "adjoint":
        n = size(17, 72)
        return _case("adjoint", "hall_periodic", n, rng.choice([2, 4]), steps=rng.randint(6, 20), checkpoint=5)
    return {"kind": "batch", "solves": rng.randint(4, 16), "draw": rng.randint(1, 10 ** 6), "nmin": 16, "nmax": 96,
            "steps": rng.randint(5, 20)}


# ---------------------------------------------------------------------------- inputs


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _nodes(c):
    return c["nx"], c["ny"], c["nz"]


def _spacing(c):
    lo, hi, periodic = DOMAINS[c["testcase"]][:3]
    return tuple((hi - lo) / (n if periodic else n - 1) for n in _nodes(c))


def _dt(c):
    """The step the testcase runs with: a CFL number for convection, dx^2 for the Hall term."""
    d = min(_spacing(c))
    return {"rotation_3D": 0.25 * d, "hall_circular_wave": 0.19 * d * d, "hall_periodic": 0.2 * d * d,
            "confined_domain": 0.2 * d * d}[c["testcase"]]


def _coords(c):
    lo, dev = DOMAINS[c["testcase"]][0], _device()
    g = [lo + torch.arange(n, dtype=torch.float64, device=dev) * d for n, d in zip(_nodes(c), _spacing(c))]
    return g[0].view(1, 1, -1), g[1].view(1, -1, 1), g[2].view(-1, 1, 1)


def _stack(c, parts):
    shape = _nodes(c)[::-1]
    return torch.stack([p.expand(shape) if torch.is_tensor(p) else torch.full(shape, float(p), dtype=torch.float64,
                                                                              device=_device()) for p in parts])


def _analytic(c, what, t=0.0):
    """b or u of the testcase on the grid, (3, nz, ny, nx)."""
    x, y, z = _coords(c)
    name = c["testcase"]
    if name == "rotation_3D":
        r3 = math.sqrt(3.0)
        if what == "u":
            return _stack(c, [(z - y) / r3 + 0 * x, (x - z) / r3 + 0 * y, (y - x) / r3 + 0 * z])
        co, s = math.cos(t), math.sin(t)
        p, q, m = 1 + 2 * co, 1 - co + r3 * s, 1 - co - r3 * s
        xx, yy, zz = (p * x + q * y + m * z) / 3, (m * x + p * y + q * z) / 3, (q * x + m * y + p * z) / 3
        al = torch.exp(-(5.0 / 3.0) * (3 - 2 * (3 + r3) * xx + 12 * xx * xx - 2 * (-3 + r3) * yy + 12 * yy * yy
                                       + 4 * r3 * zz + 12 * zz * zz))
        bx = al * (3 - r3 - 4 * r3 * yy + 4 * r3 * zz) / 48
        by = al * (-3 - r3 + 4 * r3 * xx - 4 * r3 * zz) / 48
        bz = al * (1 - 2 * xx + 2 * yy) / (8 * r3)
        return _stack(c, [(p * bx + m * by + q * bz) / 3, (q * bx + p * by + m * bz) / 3, (m * bx + q * by + p * bz) / 3])
    if name == "hall_circular_wave":
        if what == "u":
            return _stack(c, [0.0, 0.0, 0.0])
        return _stack(c, [0.1 * torch.sin(z - t), 0.1 * torch.cos(z - t), 1.0])
    if name == "hall_periodic":
        n, al, k = 0.5773502691896258, 0.5, 1.5
        co, si = ([f(k * q + al * k * t * n) for q in (x, y, z)] for f in (torch.cos, torch.sin))
        u = _stack(c, [co[1] + si[2], co[2] + si[0], co[0] + si[1]])
        return u if what == "u" else al * u + n
    px, py, pz = math.pi * x, math.pi * y, math.pi * z   # confined_domain: b and u alike
    return _stack(c, [torch.sin(px) * torch.cos(py) * torch.cos(pz), torch.cos(px) * torch.sin(py) * torch.cos(pz),
                      -2 * torch.cos(px) * torch.cos(py) * torch.sin(pz)])


def _modes(c, g, amplitude):
    """A few random long waves over the domain, in all three components."""
    lo, hi = DOMAINS[c["testcase"]][:2]
    x, y, z = ((q - lo) * (TWO_PI / (hi - lo)) for q in _coords(c))
    out = torch.zeros((3,) + _nodes(c)[::-1], dtype=torch.float64, device=_device())
    for _ in range(4):
        k = torch.randint(0, 3, (3,), generator=g).tolist()
        ph = float(torch.rand((), generator=g)) * TWO_PI
        v = (torch.randn(3, generator=g, dtype=torch.float64) * amplitude).to(_device()).view(3, 1, 1, 1)
        out += v * torch.cos(k[0] * x + k[1] * y + k[2] * z + ph)
    return out


def _inputs(c, seed):
    """The initial field of the case, (3, nz, ny, nx) in 64 bits (rounded to the case's REAL): the
    testcase's field and long waves; a thin sheet for adaptive dissipation, noise to clean."""
    g = torch.Generator().manual_seed(seed)
    b = _analytic(c, "b") + _modes(c, g, 0.02)
    if c["dissipation"] == "ADAPTIVE":
        x = _coords(c)[0]
        x0 = float(torch.rand((), generator=g)) * HALL_PERIOD
        b[1] += 0.7 * torch.tanh(torch.sin((x - x0) * 1.5) / (3.0 * _spacing(c)[0]))
    if c["kind"] in ("clean", "series"):
        gd = torch.Generator(_device()).manual_seed(seed)
        b += 1e-3 * torch.randn(b.shape, generator=gd, dtype=torch.float64, device=b.device)
    return b.float().double() if c["real"] == "float" else b


def _record(f, pad, dtype):
    """(3, nz, ny, nx) -> the reference layout (num_nodes_pad, 4)."""
    out = torch.zeros((pad, 4), dtype=dtype, device=f.device)
    out[: f[0].numel(), :3] = f.reshape(3, -1).T.to(dtype)
    return out


# ---------------------------------------------------------------------------- prepare and run


def _maps(c):
    lo, hi, periodic, hall, variable_u = DOMAINS[c["testcase"]]
    m = Maps()
    for a, n in zip("XYZ", _nodes(c)):
        m.I_Mesh.update({"NODES_" + a: n, a + "MIN": lo, a + "MAX": hi})
    m.I_TI.update({"DT": _dt(c), "time_integrator": c["integrator"]})
    for key, form in zip(("form_uibj", "form_source", "form_ujbi"), FORMS[c["forms"]]):
        m.I_IEq[key] = "USE_" + key[5:].upper() + "_" + form
    m.I_IEq["hall_term"] = "USE_HALL" if hall else "NONE"
    if c["dissipation"] != "NONE":
        m.I_IEq.update({"dissipation": "USE_ARTIFICIAL_DISSIPATION",
                        "dissipation_form": "USE_%s_DISSIPATION" % c["dissipation"]})
    m.I_DC["divergence_cleaning"] = "laplace" in c
    if "laplace" in c:
        m.I_DC["divergence_cleaning_form"] = "USE_LAPLACE_" + c["laplace"]
    m.I_Tech["REAL"] = c["real"]
    m.I_RunOps.update({"order": c["order"], "operator_form": "extended" if c["extended"] else "classical",
                       "testcase": c["testcase"], "variable_u": variable_u,
                       "periodic": "USE_PERIODIC" if periodic else "NONE"})
    return m


def prepare(case, seed):
    if case["kind"] == "batch":
        return _prepare_batch(case, seed)
    ctx = _maps(case).context()
    dtype = torch.float32 if case["real"] == "float" else torch.float64
    start = _record(_inputs(case, seed), ctx.n_pad, dtype)
    new = lambda: torch.zeros_like(start)  # noqa: E731
    s = {"case": case, "ctx": ctx, "n": ctx.n, "start": start, "b": start.clone(),
         "stream": torch.cuda.ExternalStream(ctx.stream)}
    if case["kind"] == "clean":
        return s
    s.update(u=_record(_analytic(case, "u"), ctx.n_pad, dtype), rho=torch.ones(ctx.n_pad, dtype=dtype, device="cuda"))
    if case["kind"] == "adjoint":
        g = torch.Generator().manual_seed(seed + 1)
        s["weight"] = _record(_modes(case, g, 1.0), ctx.n_pad, dtype)
        return s
    s.update(b2=new(), b3=new(), curl=new(), time=torch.zeros(2, dtype=dtype, device="cuda"))
    if case["kind"] == "list":
        s.update(names=ctx.step_kernels(), work=new(), scalar=torch.zeros(ctx.n_pad, dtype=dtype, device="cuda"))
    return s


def _rewind(s, *pairs):
    """Back to the start of the run, on the context's own stream."""
    with torch.cuda.stream(s["stream"]):
        for dst, src in pairs:
            dst.copy_(src)
        if "time" in s:
            s["time"].zero_()


def run(s):
    c, ctx = s["case"], s.get("ctx")
    n = s.get("n")
    if c["kind"] == "batch":
        s["batch"].run(c["steps"], mode="branches")
        s["batch"].unbind()
        return {"b%d" % i: f["b"] for i, f in enumerate(s["batch"].fields)}
    if c["kind"] == "clean":
        _rewind(s, (s["b"], s["start"]))
        r = ctx.clean_div(s["b"], c["max_iterations"], 1e-9, check=False)
        return {"b": s["b"][:n], "iterations": r["iterations"], "residual_norm2": r["residual_norm2"],
                "divergence_norm_initial": r["divergence_norm_initial"]}
    if c["kind"] == "adjoint":
        lam = s["b"]
        _rewind(s, (lam, s["weight"]))
        ctx.adjoint_steps(s["start"], lam, s["u"], s["rho"], c["steps"], c["checkpoint"])
        return {"gradient": lam[:n]}
    fields = (s["b"], s["b2"], s["b3"], s["curl"], s["u"], s["rho"], s["time"])
    if c["kind"] == "series":
        _rewind(s, (s["b"], s["start"]))
        r = ctx.time_steps_integrals(*fields, c["steps"], c["max_iterations"], 1e-9)
        return {"b": s["b"][:n], "time": s["time"], **r}
    if c["kind"] == "list":
        _rewind(s, (s["b"], s["start"]))
        args = fields if c["integrator"] == "SSPRK33" else fields[:2] + fields[3:]
        for _ in range(c["steps"]):
            ctx.run(s["names"], _nodes(c), *args)
        return {"b": s["b"][:n], "time": s["time"], **ctx.results(s["b"], c["steps"] * _dt(c), s["work"], s["scalar"])}
    # one solve goes on from pass to pass where it stays bounded; a forced one starts again
    if c["testcase"] in ("hall_periodic", "confined_domain"):
        _rewind(s, (s["b"], s["start"]))
    ctx.time_steps(*fields, c["steps"])
    out = {"b": s["b"][:n], "time": s["time"]}
    # the register and the curl buffer of the last stage, where the state's precision holds them
    if c["real"] == "double" and c["testcase"] == "hall_circular_wave":
        out.update(b2=s["b2"][:n], curl=s["curl"][:n])
    return out


def _prepare_batch(c, seed):
    batch = Batch(_specs(c))
    for f, spec, ctx in zip(batch.fields, _specs(c), batch.ctxs):
        b, u = _batch_fields(spec, seed)
        f["b"], f["u"] = _record(b, ctx.n_pad, torch.float64), _record(u, ctx.n_pad, torch.float64)
        f["b2"], f["b3"] = torch.zeros_like(f["b"]), torch.zeros_like(f["b"])
    torch.cuda.synchronize()
    batch.bind()
    return {"case": c, "batch": batch}


def _specs(c):
    return rotation_batch(c["solves"], c["draw"], c["nmin"], c["nmax"])


def _batch_case(spec):
    n, order = spec[:2]
    return _case("steps", "rotation_3D", (n, n, n), order)


def _gaussian(spec, t):
    """b of the rotated Gaussian bump at time t."""
    x, y, z = _coords(_batch_case(spec))
    s, co = math.sin(spec[2] * t), math.cos(spec[2] * t)
    xr, yr = co * x + s * y - 0.5, -s * x + co * y
    amp = 0.1 * 1.6487212707001282 / 1.4142135623730951 * torch.exp(-(xr * xr + yr * yr) / 0.01)
    bx, by = -2 * yr / 0.01 * amp, 2 * xr / 0.01 * amp
    return _stack(_batch_case(spec), [co * bx - s * by, s * bx + co * by, 0.0])


def _batch_fields(spec, seed):
    c = _batch_case(spec)
    x, y, z = _coords(c)
    b = _gaussian(spec, 0.0) + _modes(c, torch.Generator().manual_seed(seed + spec[0]), 0.02)
    return b, _stack(c, [-spec[2] * y, spec[2] * x, 0.0])


# ---------------------------------------------------------------------------- the work of a pass


def work(case):
    """Bytes: every field a stage, an iteration or a call combines, read once and written once,
    three components a vector field.  Operations: the stencil sums of the terms that are on."""
    if case["kind"] == "batch":
        each = [work(dict(_batch_case(s), steps=case["steps"])) for s in _specs(case)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    n = case["nx"] * case["ny"] * case["nz"]
    r = 4 if case["real"] == "float" else 8
    hall, variable_u = DOMAINS[case["testcase"]][3:]
    moving = case["testcase"] != "hall_circular_wave"
    o = case["order"]
    vec = 3 * n * r
    # a convection axis takes two vector sums, a Hall axis two scalar ones and two for the curl
    stage_flops = n * ((36 * o if moving else 0) + (24 * o if hall else 0) + 24
                       + {"NONE": 0, "HIGH_ORDER": 18 * (o + 1), "FIRST_ORDER": 45 * o, "ADAPTIVE": 120 * o}[case["dissipation"]])
    # read b (and u, rho, the register), write b (and the register)
    two = case["integrator"] == CK
    stage_bytes = 2 * vec + (2 * vec if two else 2 * vec / 3) + (vec if moving else 0) + (n * r if hall else 0)
    stages = case["steps"] * (5 if two else 3)
    # the wide Laplacian's row is 2 * order + 1 points an axis; a CG iteration reads and writes
    # the direction, the residual and the solution, and reads the Laplacian, in 64 bits
    width = 2 * o + 1 if case.get("laplace", "").startswith("WIDE") else o + 1
    cg = {"bytes": case.get("max_iterations", 0) * 7 * 8 * n + 4 * vec,
          "flops": case.get("max_iterations", 0) * (6 * width + 10) * n}
    if case["kind"] == "clean":
        return cg
    if case["kind"] == "adjoint":   # the stages twice forward, and their transposes (u at every stage)
        return {"bytes": stages * 3 * (stage_bytes + vec), "flops": stages * 4 * stage_flops}
    w = {"bytes": stages * stage_bytes, "flops": stages * stage_flops}
    if case["kind"] == "series":
        w = {k: w[k] + case["steps"] * cg[k] for k in w}
    if case["kind"] == "list":
        w["bytes"] += 3 * vec
    return w


# ---------------------------------------------------------------------------- the same in 64 bits


def _expand(tab):
    rows = [[float.fromhex(x) for x in r] for r in tab["rows"]]
    if not tab["explicit"]:
        for j in range(tab["nb"] - 1, -1, -1):
            rows.append([tab["sign"] * v for v in rows[j][::-1]])
    return np.array(rows)


class _Exact:
    """The discretisation with dense matrices along each axis; fields (3, nz, ny, nx)."""

    def __init__(self, c):
        self.c = c
        self.d, self.n = _spacing(c), _nodes(c)
        self.periodic, self.hall, self.variable_u = DOMAINS[c["testcase"]][2:]
        with open(os.path.join("inductioneq_b200", "sbp_tables.json")) as f:
            self.t = json.load(f)["%d%s" % (c["order"], "e" if c["extended"] else "c")]
        half = [float.fromhex(x) for x in self.t["Minv"]]
        self.minv = np.array(half + half[-2::-1])
        self.rows_d, self.dho = _expand(self.t["D"]), _expand(self.t["DHO"])
        self.D = [self._matrix(self.rows_d, a) / self.d[a] for a in range(3)]
        self.H = [self._dissipation(a) for a in range(3)] if c["dissipation"] == "HIGH_ORDER" else None
        self.boundary = lambda t: _analytic(c, "b", t)

    def _row(self, i, n, nb):
        return nb if self.periodic else i if i < nb else nb + (nb - (n - 1 - i) if n - 1 - i < nb else 0)

    def _to(self, m):
        return torch.tensor(m, dtype=torch.float64, device=_device())

    def _at(self, i, o, n):
        j = i + o
        return j % n if self.periodic else j if 0 <= j < n else i

    def _matrix(self, rows, a):
        n, nb, c0 = self.n[a], (len(rows) - 1) // 2, (rows.shape[1] - 1) // 2
        m = np.zeros((n, n))
        for i in range(n):
            for k, v in enumerate(rows[self._row(i, n, nb)]):
                m[i, self._at(i, k - c0, n)] += v
        return self._to(m)

    def _dissipation(self, a, start=None):
        n, nb, w = self.n[a], (len(self.dho) - 1) // 2, self.dho.shape[1]
        sign = -1.0 if (self.c["order"] // 2 + 1) % 2 else 1.0
        m = np.zeros((n, n))
        for i in range(n):
            r = self._row(i, n, nb)
            for s in range(-w + 1, 1) if start is None else (start,):
                for k in range(w):
                    m[i, self._at(i, s + k, n)] += sign * self.minv[r] * self.dho[r, s + w - 1] * self.dho[nb, k]
        return self._to(m)

    @staticmethod
    def along(m, f, a):
        if a == 0:
            return f @ m.T
        if a == 1:
            return m @ f
        return (m @ f.reshape(f.shape[:-3] + (f.shape[-3], -1))).reshape(f.shape)

    def curl(self, b):
        d = lambda a, k: self.along(self.D[a], b[k], a)  # noqa: E731
        return torch.stack([d(1, 2) - d(2, 1), d(2, 0) - d(0, 2), d(0, 1) - d(1, 0)])

    def div(self, b):
        return sum(self.along(self.D[a], b[a], a) for a in range(3))

    def volume(self, b, u):
        """2 sum_k D F of the three flux forms, expanded (the row sums of D are zero)."""
        f1, f2, f3 = FORMS[self.c["forms"]]
        w = dict.fromkeys("abcdef", 0.0)   # D(u Ba), Ba D(u), u D(Ba), D(ua B), ua D(B), B D(ua)
        for k, v in {"CENTRAL": {"a": 1}, "SPLIT": {"a": .5, "b": .5, "c": .5}, "PRODUCT": {"b": 1, "c": 1}}[f1].items():
            w[k] += v
        for k, v in {"ZERO": {}, "CENTRAL": {"c": 1}, "SPLIT": {"c": .5, "a": .5, "b": -.5}}[f2].items():
            w[k] -= v
        for k, v in {"CENTRAL": {"d": 1}, "SPLIT": {"d": .5, "e": .5, "f": .5}, "PRODUCT": {"e": 1, "f": 1}}[f3].items():
            w[k] -= v
        out = torch.zeros_like(b)
        for a in range(3):
            D = lambda f: self.along(self.D[a], f, a)  # noqa: B023, E731
            if w["a"]:
                out = out + w["a"] * D(u * b[a])
            if w["b"]:
                out = out + w["b"] * b[a] * D(u)
            if w["c"]:
                out = out + w["c"] * u * D(b[a])
            if w["d"]:
                out = out + w["d"] * D(u[a] * b)
            if w["e"]:
                out = out + w["e"] * u[a] * D(b)
            if w["f"]:
                out = out + w["f"] * b * D(u[a])
        return out

    def _faces(self, a):
        left = torch.zeros(self.n[a], dtype=torch.float64, device=_device())
        right = left.clone()
        left[0], right[-1] = 1.0, 1.0
        shape = [1, 1, 1]
        shape[2 - a] = -1
        return left.view(shape), right.view(shape)

    def surface(self, b, J, u, t):
        if self.periodic:
            return 0.0
        out = torch.zeros_like(b)
        diff = None if self.hall else b - self.boundary(t)
        for a in range(3):
            left, right = self._faces(a)
            s = self.minv[0] / self.d[a]
            if self.hall:
                tv = 0.5 * u[a] - J[a]
                c1 = right * (tv < 0) - left * (tv > 0)
                out = out + s * (c1 * tv * b + (right - left) * b[a] * J)
            else:
                out = out + s * (right * (u[a] < 0) - left * (u[a] > 0)) * u[a] * diff
        return out

    def _shift(self, f, a, o):
        idx = torch.tensor([self._at(i, o, self.n[a]) for i in range(self.n[a])], device=f.device)
        return f.index_select(f.dim() - 1 - a, idx)

    def _kappa(self, k, a, b1, b2, u1, u2):
        """The switch between the first-order and the high-order form (MP2 1 .. 10, C 1 .. 10)."""
        s = torch.maximum(u1.abs(), u2.abs()) * (b1 - b2) ** 2
        kk = max(k, 1) ** 2
        lo, hi = kk * self.d[a], kk * 100.0 * self.d[a]
        return torch.where(s >= hi, 1.0, torch.where(s > lo, ((s - lo).clamp_min(0) / (hi - lo)).sqrt(), 0.0))

    def dissipation(self, b, u):
        form = self.c["dissipation"]
        if form == "NONE":
            return 0.0
        if form == "HIGH_ORDER":
            return sum(self.along(self.H[a], b, a) for a in range(3))
        out = torch.zeros_like(b)
        nb, c0 = (len(self.rows_d) - 1) // 2, (self.rows_d.shape[1] - 1) // 2
        for a in range(3):
            for k in range(self.rows_d.shape[1]):
                co = np.array([abs(self.rows_d[self._row(i, self.n[a], nb), k]) for i in range(self.n[a])])
                if not co.any():
                    continue
                shape = [1, 1, 1]
                shape[2 - a] = -1
                bk, uk = self._shift(b, a, k - c0), self._shift(u, a, k - c0)
                wt = self._to(co).view(shape) / self.d[a] * torch.maximum(uk.abs(), u.abs())
                if form == "ADAPTIVE":
                    wt = wt * self._kappa(abs(k - c0), a, bk, b, uk, u)
                out = out + wt * (bk - b)
            if form == "ADAPTIVE":
                w = self.dho.shape[1]
                for s in range(-w + 1, 1):
                    e1, e2 = s + w - 1, s + w - 2
                    k1 = self._kappa(1, a, self._shift(b, a, e1), self._shift(b, a, e2), self._shift(u, a, e1),
                                     self._shift(u, a, e2))
                    out = out + (1 - k1) * self.along(self._dissipation(a, s), b, a)
        return out

    def rhs(self, b, u, t):
        J = self.curl(b) if self.hall else None
        db = self.volume(b, u) + self.surface(b, J, u, t)
        if self.hall:
            db = db + sum(self.along(self.D[a], J[a] * b - J * b[a], a) for a in range(3))
        return db + self.dissipation(b, u)

    def steps(self, b, u, dt, count, t=0.0):
        """Returns b, the time, and the register and curl(b) of the last stage."""
        at = (lambda s: _analytic(self.c, "u", s)) if self.variable_u else lambda s: u
        reg = cu = None
        for _ in range(count):
            if self.c["integrator"] == CK:
                for s, (A, B, C) in enumerate(CK_TABLE):
                    cu = b
                    k = dt * self.rhs(b, at(t + C * dt), t + C * dt)
                    reg = k if s == 0 else A * reg + k
                    b = b + B * reg
            else:
                b2 = b + dt * self.rhs(b, at(t), t)
                b3 = 0.75 * b + 0.25 * (b2 + dt * self.rhs(b2, at(t + dt), t + dt))
                b = b / 3 + 2.0 / 3.0 * (b3 + dt * self.rhs(b3, at(t + 0.5 * dt), t + 0.5 * dt))
            t = t + dt
        return b, t, reg, cu

    def clean(self, b, cap):
        """Conjugate gradients on (-Laplace) phi = div b inside one layer, then the projection."""
        key = {"WIDE_STENCIL_DIRICHLET": "WS_D0", "NARROW_STENCIL_DIRICHLET": "NS_D0"}[self.c["laplace"]]
        rows = _expand(self.t["laplace"][key])
        L = [self._matrix(rows, a) / self.d[a] ** 2 for a in range(3)]
        inner = torch.zeros_like(b[0])
        inner[1:-1, 1:-1, 1:-1] = 1.0
        r = self.div(b) * inner
        phi, p = torch.zeros_like(r), torch.zeros_like(r)
        rr = (r * r).sum()
        first, old = rr.sqrt(), torch.ones_like(rr)
        for _ in range(cap):
            p = rr / old * p + r
            q = sum(self.along(L[a], p, a) for a in range(3)) * inner
            alpha = rr / (p * q).sum()
            phi, r = phi + alpha * p, r - alpha * q
            old, rr = rr, (r * r).sum()
        return b + torch.stack([self.along(self.D[a], phi, a) for a in range(3)]), rr, first

    def norm2(self, f):
        w = 1.0
        for a in range(3):
            nb = (len(self.minv) - 1) // 2
            shape = [1, 1, 1]
            shape[2 - a] = -1
            w = w * self._to([self.d[a] / self.minv[self._row(i, self.n[a], nb)] for i in range(self.n[a])]).view(shape)
        return float((w * f * f).sum())

    def diagnostics(self, b, t):
        return self.norm2(b), math.sqrt(self.norm2(self.div(b))), math.sqrt(self.norm2(b - _analytic(self.c, "b", t)))


# CarpenterKennedy2N54: register factor, weight, stage time
CK_TABLE = (
    (0.0, 1432997174477.0 / 9575080441755.0, 0.0),
    (-567301805773.0 / 1357537059087.0, 5161836677717.0 / 13612068292357.0, 1432997174477.0 / 9575080441755.0),
    (-2404267990393.0 / 2016746695238.0, 1720146321549.0 / 2090206949498.0, 2526269341429.0 / 6820363962896.0),
    (-3550918686646.0 / 2091501179385.0, 3134564353537.0 / 4481467310338.0, 2006345519317.0 / 3224310063776.0),
    (-1275806237668.0 / 842570457699.0, 2277821191437.0 / 14882151754819.0, 2802321613138.0 / 2924317926251.0))


def exact(case, seed):
    if case["kind"] == "batch":
        out = {}
        for i, spec in enumerate(_specs(case)):
            b, u = _batch_fields(spec, seed)
            e = _Exact(_batch_case(spec))
            e.boundary = lambda t, spec=spec: _gaussian(spec, t)
            out["b%d" % i] = _record(e.steps(b, u, spec[3], case["steps"])[0], b[0].numel(), torch.float64)
        return out
    e = _Exact(case)
    b, n, dt = _inputs(case, seed), case["nx"] * case["ny"] * case["nz"], _dt(case)
    rec = lambda f: _record(f, n, torch.float64)  # noqa: E731
    if case["kind"] == "clean":
        b, rr, first = e.clean(b, case["max_iterations"])
        return {"b": rec(b), "iterations": None, "residual_norm2": float(rr), "divergence_norm_initial": float(first)}
    u = _analytic(case, "u")
    if case["real"] == "float":
        u = u.float().double()
    if case["kind"] == "adjoint":
        w = _modes(case, torch.Generator().manual_seed(seed + 1), 1.0)
        b.requires_grad_(True)
        (e.steps(b, u, dt, case["steps"])[0] * w).sum().backward()
        return {"gradient": rec(b.grad)}
    if case["kind"] == "series":
        t, rows = 0.0, []
        for _ in range(case["steps"]):
            rows.append(e.diagnostics(b, t))
            b, t = e.steps(b, u, dt, 1, t)[:2]
            b = e.clean(b, case["max_iterations"])[0]
        en, dv, l2 = np.array(rows).T
        return {"b": rec(b), "time": torch.full((2,), t, dtype=torch.float64), "energy": en, "divergence_norm": dv,
                "l2_error": l2}
    b, t, reg, last = e.steps(b, u, dt, case["steps"])
    out = {"b": rec(b), "time": torch.full((2,), t, dtype=torch.float64)}
    if case["kind"] == "list":
        en, dv, l2 = e.diagnostics(b, t)
        out.update(abs_err=l2, rel_err=l2 / math.sqrt(e.norm2(_analytic(case, "b", t))), divergence_norm=dv, energy=en)
    elif case["real"] == "double" and case["testcase"] == "hall_circular_wave":
        out.update(b2=rec(reg), curl=rec(e.curl(last)))
    return out
