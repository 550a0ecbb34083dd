"""What a program does with this framework, as cases that can be timed.

A case is one call (or one short sequence of calls) through the public Python entry points,
which are thin ctypes wrappers of the C ABI.  Kinds:

* ``solve``   -- a batch of nonlinear samples on one geometry (``Plan.solve_device`` with
  device buffers, or ``Plan.solve`` with host buffers), on the planar square, the
  rotor-stator sector or the axisymmetric plunger, in the plain FP64 form or an accelerated
  one;
* ``meshes``  -- one sample on each of several geometries of uneven size (``Multi.solve``);
* ``csr``     -- one linear system already in device memory (``csr_pcg_noalloc``);
* ``tangent`` -- circuit derivatives at an operating point (``Plan.solve_tangent``);
* ``post``    -- force, torque and air-gap samples of solved fields in device memory
  (``Postprocess.compute_device``);
* ``network`` -- the warm start's network: the forward and backward pass of one training
  batch (``Mlp.loss_gradient``), or inference (``Mlp.forward``).

The geometry of a case is fixed by its sizes, as the mesh file of a program is; currents,
magnet angles, coercivities, fields and network data come from the seed.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "femm-gpu_b200"))

import femm_gpu_b200 as fg  # noqa: E402
from femm_gpu_b200 import learned, meshes  # noqa: E402
from femm_gpu_b200.capi import csr_pcg_noalloc  # noqa: E402

DEVICE = "cuda"
ANGLES = 45  # air-gap probes of a sector

# Plan options of the forms a program can ask for.
FORMS = {
    "plain": {},
    "block8": dict(preconditioner=1, block_size=8),
    "mixed": dict(precision=1),
    "fast8": dict(precision=1, preconditioner=1, block_size=8, from_iterate=True),
    "fast32": dict(precision=1, preconditioner=1, block_size=32, from_iterate=True),
}


def listed():
    return [
        # A small linear system handed over in device memory: latency of one call.
        dict(name="csr_4k", kind="csr", size=64),
        # One sample on a small mesh: a design loop's single evaluation.
        dict(name="solve_4k_x1", kind="solve", mesh="square", size=64, items=1, form="plain", host=False),
        # A chunk of 32 samples of a saturated machine sector (anti-periodic edges): many
        # relaxed Newton steps on a mid-size operator.
        dict(name="sector_10k_x32", kind="solve", mesh="sector", size=80, items=32, form="plain", host=False),
        # The 40k-node sector with a ragged batch (5 of 8 lanes in use).
        dict(name="sector_40k_x5", kind="solve", mesh="sector", size=160, items=5, form="plain", host=False),
        # The planar nonlinear workload of the benchmark: 251k nodes, 8 samples.
        dict(name="solve_251k_x8", kind="solve", mesh="square", size=500, items=8, form="plain", host=False),
        # The same workload in the fast form (FP32 inner solves, 8-row blocks, from the iterate).
        dict(name="fast_251k_x8", kind="solve", mesh="square", size=500, items=8, form="fast8", host=False),
        # One sample at a million nodes, FP32 inner solves with 32-row blocks.
        dict(name="fast_1m_x1", kind="solve", mesh="square", size=1000, items=1, form="fast32", host=False),
        # Axisymmetric training solves for the warm start, through host buffers.
        dict(name="plunger_25k_x32_host", kind="solve", mesh="plunger", size=111, items=32, form="plain", host=True),
        # One sample on each of 12 meshes of uneven size in one launch per Newton step.
        dict(name="meshes_x12", kind="meshes", count=12, low=3000, high=40000),
        # Differential inductances of a machine: three directions at one operating point.
        dict(name="tangent_40k_x3", kind="tangent", size=160, items=3),
        # Torque, force and 45 air-gap samples of 32 solved fields.
        dict(name="post_40k_x32", kind="post", size=160, items=32),
        # Forward and backward pass of one training batch of the warm start's network.
        dict(name="network_256", kind="network", op="gradient", batch=256, hidden=256, outputs=64),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "meshes", "csr", "tangent", "post", "network"])
    if kind == "solve":
        mesh = rng.choice(["square", "square", "sector", "plunger"])
        form = rng.choice(["plain", "plain", "plain", "block8", "mixed", "fast8"])
        size = {"square": _log_int(rng, 24, 400), "sector": _log_int(rng, 20, 160),
                "plunger": _log_int(rng, 24, 223)}[mesh]
        case = dict(kind="solve", mesh=mesh, size=size, items=_log_int(rng, 1, 32), form=form,
                    host=rng.random() < 0.3)
        while case["items"] > 1 and _seconds(case) > 0.3:
            case["items"] = case["items"] * 2 // 3
        return case
    if kind == "meshes":
        low = _log_int(rng, 1000, 8000)
        return dict(kind="meshes", count=rng.randint(2, 16), low=low, high=_log_int(rng, 2 * low, 40000))
    if kind == "csr":
        return dict(kind="csr", size=_log_int(rng, 8, 120))
    if kind in ("tangent", "post"):
        items = rng.randint(1, 8) if kind == "tangent" else rng.randint(1, 32)
        return dict(kind=kind, size=_log_int(rng, 20, 160), items=items)
    op = rng.choice(["gradient", "gradient", "forward"])
    return dict(kind="network", op=op, batch=_log_int(rng, 16, 1024 if op == "gradient" else 4096),
                hidden=_log_int(rng, 48, 320), outputs=_log_int(rng, 8, 96))


# ---------------------------------------------------------------------------------------
# Geometry and inputs
# ---------------------------------------------------------------------------------------

LIMIT_A = {"square": 20.0, "sector": 15.0, "plunger": 30.0}  # current range of each mesh


@functools.lru_cache(maxsize=4)
def _mesh(mesh, size):
    if mesh == "square":
        return meshes.square_nonlinear(size, seed=2)
    if mesh == "sector":
        m = meshes.annular_sector(size, max(8, size * 25 // 16))
        m.group = np.array([0, 10, 10, 3, 4, 5, 6], np.int32)  # rotor iron and magnets: group 10
        return m
    return meshes.axisymmetric_plunger(size, 2 * size + 1)


def _model(mesh, size, rng):
    """The geometry with this seed's magnet angle."""
    m = _mesh(mesh, size)
    m = fg.Model(**{f: getattr(m, f) for f in m.__dataclass_fields__})
    if mesh == "square":
        m.mag_deg = np.array(m.mag_deg)
        m.mag_deg[2] = rng.uniform(0.0, 360.0)
    return m


def _samples(case, rng, circuits):
    cur = rng.uniform(-1.0, 1.0, size=(case["items"], circuits)) * LIMIT_A[case["mesh"]]
    hc = rng.uniform(8.5e5, 9.5e5, size=case["items"]) / 9.0e5 if case["mesh"] == "sector" else None
    return cur, hc


def _solve_inputs(case, seed):
    rng = np.random.default_rng(seed)
    model = _model(case["mesh"], case["size"], rng)
    return (model, *_samples(case, rng, model.circuit_count))


def _meshes_inputs(case, seed):
    rng = np.random.default_rng(seed)
    nodes = np.exp(np.linspace(math.log(case["low"]), math.log(case["high"]), case["count"]))
    out = []
    for i, n in enumerate(nodes):
        m = max(8, int(round(math.sqrt(n))) - 1)
        model = meshes.square_nonlinear(m, seed=100 + i, magnet_deg=float(rng.uniform(0.0, 360.0)))
        out.append((model, rng.uniform(-20.0, 20.0, size=3)))
    return out


def _csr_inputs(case, seed):
    rng = np.random.default_rng(seed)
    return _model("square", case["size"], rng), rng.uniform(-20.0, 20.0, size=3)


def _field_options(steps):
    """Options of a solve stopped after a few Newton steps: fields near a solution."""
    return fg.production_options(max_newton_iterations=steps, recover_nonconvergence=0)


def _sector_fields(plan, size, items, seed, steps):
    rng = np.random.default_rng(seed)
    cur, hc = _samples(dict(mesh="sector", items=items), rng, plan.C)
    out = [torch.zeros((items, w), dtype=torch.float64, device=DEVICE) for w in (plan.N, plan.E, plan.E)]
    dev = [torch.tensor(x, device=DEVICE) for x in (cur, hc)]
    torch.cuda.synchronize()
    plan.solve_device(items, dev[0].data_ptr(), options=_field_options(steps), hc_ptr=dev[1].data_ptr(),
                      a_ptr=out[0].data_ptr(), b1_ptr=out[1].data_ptr(), b2_ptr=out[2].data_ptr())
    torch.cuda.synchronize()
    return cur, hc, out


def _rotor_mask(model):
    """Selector of the weighted-stress force: 1 on and inside the magnets, 0 from mid-gap."""
    return (np.hypot(model.xy[:, 0], model.xy[:, 1]) < 0.0452).astype(np.float64)


def _network_inputs(case, seed):
    rng = np.random.default_rng(seed)
    h, o = case["hidden"], case["outputs"]
    x = rng.normal(size=(case["batch"], 4)).astype(np.float32)
    t = rng.normal(size=(case["batch"], o)).astype(np.float32)
    p = np.concatenate([rng.uniform(-1.0, 1.0, size=n).astype(np.float32) / np.float32(math.sqrt(f))
                        for n, f in ((h * 4, 4), (h, 4), (h * h, h), (h, h), (o * h, h), (o, h))])
    return x, t, p


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "solve":
        model, cur, hc = _solve_inputs(case, seed)
        plan = s["plan"] = fg.Plan(model, **FORMS[case["form"]])
        k, s["cur"], s["hc"] = case["items"], cur, hc
        if not case["host"]:
            s["dev"] = [None if x is None else torch.tensor(x, device=DEVICE) for x in (cur, hc)]
            s["out"] = [torch.zeros((k, w), dtype=torch.float64, device=DEVICE)
                        for w in (plan.N, plan.E, plan.E, plan.C)]
        else:
            s["buffers"] = None
    elif kind == "meshes":
        inputs = _meshes_inputs(case, seed)
        s["plans"] = [fg.Plan(m) for m, _ in inputs]
        s["multi"] = fg.Multi(s["plans"])
        s["cur"] = [c for _, c in inputs]
    elif kind == "csr":
        model, cur = _csr_inputs(case, seed)
        plan = fg.Plan(model)
        ro, col, _, _, _ = plan.symbolic()
        vals, diag, rhs = plan.assemble(np.zeros(plan.N), cur, 0)
        s["n"] = plan.rows
        s["dev"] = [torch.tensor(x, device=DEVICE) for x in (ro, col, vals[0], diag[0], rhs[0])]
        s["x"] = torch.zeros(plan.rows, dtype=torch.float64, device=DEVICE)
        plan.close()
    elif kind == "tangent":
        plan = s["plan"] = fg.Plan(_mesh("sector", case["size"]))
        cur, _, out = _sector_fields(plan, case["size"], 1, seed, 6)
        s["base"], s["cur"] = out[0][0].cpu().numpy(), cur[0]
        s["directions"] = np.random.default_rng(seed + 1).normal(size=(case["items"], plan.C))
    elif kind == "post":
        model = _mesh("sector", case["size"])
        plan = s["plan"] = fg.Plan(model)
        s["fields"] = _sector_fields(plan, case["size"], case["items"], seed, 2)[2]
        s["post"] = fg.Postprocess(plan, selected_group=10, air_group=0, radius_m=0.0455,
                                   angles_rad=np.radians(np.linspace(1.0, 89.0, ANGLES)), mask=_rotor_mask(model))
    else:
        s["x"], s["t"], p = _network_inputs(case, seed)
        s["mlp"] = learned.Mlp(4, case["hidden"], case["outputs"])
        s["mlp"].set_parameters(p)
    return s


def _counts(info):
    return np.array([i.status for i in info]), np.array([i.iterations for i in info])


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "solve" and not case["host"]:
        (cur, hc), (a, b1, b2, flux) = s["dev"], s["out"]
        info = s["plan"].solve_device(case["items"], cur.data_ptr(), hc_ptr=None if hc is None else hc.data_ptr(),
                                      a_ptr=a.data_ptr(), b1_ptr=b1.data_ptr(), b2_ptr=b2.data_ptr(),
                                      flux_ptr=flux.data_ptr())
        status, newton = _counts(info)
        return {"a": a, "b1": b1, "b2": b2, "flux": flux, "status": status, "newton": newton}
    if kind == "solve":
        r = s["buffers"] = s["plan"].solve(s["cur"], hc_scale=s["hc"], out=s["buffers"])
        status, newton = _counts(r.info)
        return {"a": r.a, "b1": r.b1, "b2": r.b2, "flux": r.flux, "status": status, "newton": newton}
    if kind == "meshes":
        a, b1, b2, flux, info = s["multi"].solve(s["cur"])
        status, newton = _counts(info)
        return {"a": np.concatenate(a), "b1": np.concatenate(b1), "b2": np.concatenate(b2),
                "flux": np.concatenate(flux), "status": status, "newton": newton}
    if kind == "csr":
        status, info = csr_pcg_noalloc(s["n"], *[t.data_ptr() for t in s["dev"]], s["x"].data_ptr())
        return {"x": s["x"], "status": np.array([status, info.status])}
    if kind == "tangent":
        da, db1, db2, dflux, info = s["plan"].solve_tangent(s["base"], s["cur"], s["directions"])
        return {"da": da, "db1": db1, "db2": db2, "dflux": dflux, "status": np.array([i.status for i in info])}
    if kind == "post":
        r = s["post"].compute_device(case["items"], *[t.data_ptr() for t in s["fields"]])
        return {"force": r.force, "torque": r.torque, "radial_b": r.radial_b, "status": r.status}
    if case["op"] == "forward":
        return {"y": s["mlp"].forward(s["x"])}
    loss, grad = s["mlp"].loss_gradient(s["x"], s["t"])
    return {"loss": loss, "gradient": grad}


# ---------------------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------------------

# CG iterations of a whole solve over the mesh size (nodes along one side, or radially).
ITERATIONS = {"square": 13.3, "sector": 205.0, "plunger": 18.4}
SHARE = {"plain": 1.0, "block8": 0.72, "mixed": 1.0, "fast8": 0.39, "fast32": 0.35}  # of the plain form's


def _nodes(mesh, size):
    if mesh == "square":
        return (size + 1) ** 2
    if mesh == "sector":
        return (size + 1) * (max(8, size * 25 // 16) + 1)
    return (size + 1) * (2 * size + 2)


def _cg(nodes, items, iterations, word=8):
    """One CG iteration reads the operator (7 entries a row) and reads and writes the
    iterate, the residual and the direction once; each entry is a multiply and an add."""
    return {"bytes": iterations * (items * nodes * (7 + 6) * word + 28 * nodes),
            "flops": iterations * items * nodes * (2 * 7 + 2 * 6)}


def _seconds(case):
    """Rough time of a plain solve, to keep drawn cases below the largest listed one."""
    n = _nodes(case["mesh"], case["size"]) * case["items"]
    return ITERATIONS[case["mesh"]] * case["size"] * (1.2e-5 + 3.2e-11 * n)


def work(case):
    kind = case["kind"]
    if kind == "solve":
        nodes = _nodes(case["mesh"], case["size"])
        form = case["form"]
        its = ITERATIONS[case["mesh"]] * case["size"] * SHARE[form]
        return _cg(nodes, case["items"], its, 8 if form in ("plain", "block8") else 4)
    if kind == "meshes":
        total = {"bytes": 0.0, "flops": 0.0}
        for n in np.exp(np.linspace(math.log(case["low"]), math.log(case["high"]), case["count"])):
            for key, v in _cg(float(n), 1, 13.3 * math.sqrt(n)).items():
                total[key] += v
        return total
    if kind == "csr":
        return _cg(case["size"] ** 2, 1, 4.0 * case["size"])
    nodes = _nodes("sector", case.get("size", 0))
    k = case.get("items", 1)
    if kind == "tangent":  # one operator for all directions
        its = 7.6 * case["size"]
        return {"bytes": its * nodes * (7 * 8 + 28 + 48 * k), "flops": its * k * nodes * 26}
    if kind == "post":  # five geometry words and two field words per element
        return {"bytes": 2 * nodes * (40 + 16 * k), "flops": 2 * nodes * k * 24}
    b, h, o = case["batch"], case["hidden"], case["outputs"]
    params = 5 * h + h * h + h + o * h + o
    passes = 3 if case["op"] == "gradient" else 1
    return {"bytes": 4 * (params * (2 if passes == 3 else 1) + b * (4 + o)),
            "flops": passes * 2 * b * (4 * h + h * h + h * o)}


# ---------------------------------------------------------------------------------------
# The same results in 64 bits: plain torch, solved to rounding
# ---------------------------------------------------------------------------------------

BARY = [(1 / 3, 1 / 3, 1 / 3)] + [p for w in ((0.059715871789770, 0.470142064105115),
                                              (0.797426985353087, 0.101286507323456))
                                  for p in ((w[0], w[1], w[1]), (w[1], w[0], w[1]), (w[1], w[1], w[0]))]
WEIGHT = [0.225] + [0.132394152788506] * 3 + [0.125939180544827] * 3


def _spline(b, h):
    """FEMM's DC B-H curve: cubic with continuous second derivative (natural ends), the
    table smoothed by three-point means until every segment is monotone."""
    b, h = np.array(b, float), np.array(h, float)
    n = b.size
    while True:
        m, rhs = np.zeros((n, n)), np.zeros(n)
        for i in range(n):
            for lo, hi in ((i - 1, i), (i, i + 1)):
                if 0 <= lo and hi < n:
                    d = b[hi] - b[lo]
                    m[i, i] += 4 / d
                    m[i, lo if hi == i else hi] += 2 / d
                    rhs[i] += 6 * (h[hi] - h[lo]) / d ** 2
        s = np.linalg.solve(m, rhs)
        ok = True
        for i in range(n - 1):
            d, dh = b[i + 1] - b[i], h[i + 1] - h[i]
            c = (3 * (d * (s[i] + s[i + 1]) - 2 * dh) / d ** 3, -2 * (2 * d * s[i] + d * s[i + 1] - 3 * dh) / d ** 2, s[i])
            roots = np.roots(np.trim_zeros(c, "f")) if any(c[:2]) else np.array([])
            ok = ok and not any(abs(r.imag) == 0 and 0 <= r.real <= d for r in np.atleast_1d(roots))
        if ok:
            return b, h, s
        b[1:-1], h[1:-1] = ((v[:-2] + v[1:-1] + v[2:]) / 3 for v in (b.copy(), h.copy()))


class _Fem:
    """P1 magnetostatics on one model, all samples of a batch side by side ([..., k])."""

    def __init__(self, m):
        t = lambda x, d=torch.float64: torch.as_tensor(np.ascontiguousarray(x), device=DEVICE).to(d)  # noqa: E731
        self.m, self.tri, mat = m, t(m.tri, torch.long), t(m.tri_mat, torch.long)
        self.N, self.axi = m.node_count, m.problem_type == fg.AXISYMMETRIC
        p = t(m.xy)[self.tri]
        x, y = p[..., 0], p[..., 1]
        det = (x[:, 1] - x[:, 0]) * (y[:, 2] - y[:, 0]) - (x[:, 2] - x[:, 0]) * (y[:, 1] - y[:, 0])
        dx = torch.stack([y[:, 1] - y[:, 2], y[:, 2] - y[:, 0], y[:, 0] - y[:, 1]], 1) / det[:, None]
        dy = torch.stack([x[:, 2] - x[:, 1], x[:, 0] - x[:, 2], x[:, 1] - x[:, 0]], 1) / det[:, None]
        area = det / 2
        # Quadrature points: weight, shape values and the two components of B per nodal A.
        self.points = []
        if self.axi:
            for bary, w in zip(BARY, WEIGHT):
                n = torch.tensor(bary, device=DEVICE, dtype=torch.float64)
                r = x @ n
                self.points.append((2 * math.pi * r * area * w, n.expand(len(area), 3), -dy, dx + n / r[:, None]))
            third = torch.full((3,), 1 / 3, device=DEVICE, dtype=torch.float64)
            self.centre = (-dy, dx + third / (x @ third)[:, None])
        else:
            self.points.append((area, torch.full_like(dx, 1 / 3), dy, -dx))
            self.centre = (dy, -dx)
        self.mat, self.area, self.cen = mat, area, (x.mean(1), y.mean(1))
        self.nu0, self.alpha, self.jpa = t(m.nu0)[mat], t(m.alpha)[mat], t(m.j_per_a)[mat]
        self.circuit = t(m.circuit_index, torch.long)[mat]
        self.curve = t(m.curve_index, torch.long)[mat]
        self.curves = [tuple(t(v) for v in _spline(b, h)) for b, h in m.curves]
        # Signed folding of the constraint pairs (they share no node), fixed nodes removed.
        root, sign = np.arange(self.N), np.ones(self.N)
        root[m.con_b], sign[m.con_b] = m.con_a, m.con_sign
        free = root == np.arange(self.N)
        free[m.dir_nodes] = False
        row = np.full(self.N, -1)
        row[free] = np.arange(free.sum())
        fixed = np.zeros(self.N, bool)
        fixed[m.dir_nodes] = True
        row = np.where(fixed[root] | fixed, -1, row[root])
        self.n, self.row, self.sign = int(free.sum()), t(row, torch.long), t(sign)
        er, es = self.row[self.tri], self.sign[self.tri]
        pair = (er[:, :, None] >= 0) & (er[:, None, :] >= 0)
        self.keep = pair.reshape(-1).nonzero()[:, 0]
        self.pair_sign = (es[:, :, None] * es[:, None, :]).reshape(-1)[self.keep, None]
        key = (er[:, :, None] * self.n + er[:, None, :]).reshape(-1)[self.keep]
        uniq, inv = torch.unique(key, return_inverse=True)
        r, c = uniq // self.n, uniq % self.n
        count = torch.bincount(r, minlength=self.n)
        self.W = int(count.max())
        at = r * self.W + torch.arange(len(r), device=DEVICE) - (torch.cumsum(count, 0) - count)[r]
        self.slot = at[inv]
        self.col = torch.zeros(self.n * self.W, dtype=torch.long, device=DEVICE)
        self.col[at] = c
        self.diag = at[r == c]
        # Loads: magnets and, per ampere, each circuit.
        th = np.radians(m.mag_deg)
        hx, hy = t(m.hc * np.cos(th))[mat], t(m.hc * np.sin(th))[mat]
        self.magnet = self._load(sum(w[:, None] * (hx[:, None] * bx + hy[:, None] * by)
                                     for w, _, bx, by in self.points)[..., None])[:, 0]
        coil = sum(w[:, None] * self.jpa[:, None] * s for w, s, _, _ in self.points)
        on = torch.stack([self.circuit == i for i in range(m.circuit_count)], -1)
        self.coil_elements = coil[..., None] * on[:, None, :]
        self.coils = self._load(self.coil_elements)

    def _load(self, v):  # [E, 3, k] -> [n, k]
        er = self.row[self.tri].reshape(-1)
        ok = er >= 0
        v = (v * self.sign[self.tri][..., None]).reshape(-1, v.shape[-1])
        return torch.zeros((self.n, v.shape[-1]), dtype=torch.float64, device=DEVICE).index_add_(0, er[ok], v[ok])

    def nodal(self, x):
        a = x[self.row.clamp(min=0)] * self.sign[:, None]
        return torch.where((self.row >= 0)[:, None], a, torch.zeros_like(a))  # fixed nodes are at 0

    def _nu(self, b):
        nu = self.nu0[:, None] * (1 + self.alpha[:, None] * b * b)
        dnu = (self.nu0 * self.alpha)[:, None].expand_as(b).clone()
        for i, (kb, kh, ks) in enumerate(self.curves):
            e = (self.curve == i).nonzero()[:, 0]
            v = b[e]
            j = torch.searchsorted(kb, v.contiguous()).clamp(1, len(kb) - 1)
            lo, d = kb[j - 1], kb[j] - kb[j - 1]
            z = (v - lo) / d
            h = ((1 - 3 * z ** 2 + 2 * z ** 3) * kh[j - 1] + z * (1 - z) ** 2 * d * ks[j - 1]
                 + z ** 2 * (3 - 2 * z) * kh[j] + z ** 2 * (z - 1) * d * ks[j])
            dh = (6 * z * (z - 1) * (kh[j - 1] - kh[j]) / d + (1 - 4 * z + 3 * z ** 2) * ks[j - 1]
                  + z * (3 * z - 2) * ks[j])
            over = v > kb[-1]
            h, dh = torch.where(over, kh[-1] + ks[-1] * (v - kb[-1]), h), torch.where(over, ks[-1].expand_as(v), dh)
            zero = v < 1e-12
            s = torch.where(zero, torch.ones_like(v), v)
            nu[e] = torch.where(zero, ks[0].expand_as(v), h / s)
            dnu[e] = torch.where(zero, torch.zeros_like(v), 0.5 * (dh / s ** 2 - h / s ** 3))
        return nu, dnu

    def system(self, x, jacobian):
        """K(A) A, and the Jacobian's entries as [n * W, k]."""
        a = self.nodal(x)[self.tri]
        f, mats = 0, 0
        for w, _, bx, by in self.points:
            B1, B2 = ((a * v[..., None]).sum(1) for v in (bx, by))
            nu, dnu = self._nu(torch.hypot(B1, B2))
            bd = B1[:, None] * bx[..., None] + B2[:, None] * by[..., None]
            f = f + (w[:, None] * nu)[:, None] * bd
            if jacobian:
                g = bx[:, :, None] * bx[:, None, :] + by[:, :, None] * by[:, None, :]
                mats = mats + (w[:, None] * nu)[:, None, None] * g[..., None]
                mats = mats + (2 * w[:, None] * dnu)[:, None, None] * bd[:, :, None] * bd[:, None, :]
        values = None
        if jacobian:
            values = torch.zeros((self.n * self.W, x.shape[1]), dtype=torch.float64, device=DEVICE)
            values.index_add_(0, self.slot, mats.reshape(-1, x.shape[1])[self.keep] * self.pair_sign)
        return self._load(f), values

    def times(self, values, x):
        return (values.view(self.n, self.W, -1) * x[self.col].view(self.n, self.W, -1)).sum(1)

    def cg(self, values, b, tol, most=30000):
        inv = 1 / values[self.diag]
        x, r = torch.zeros_like(b), b.clone()
        z = inv * r
        p, rz, stop = z, (r * z).sum(0), tol * b.norm(dim=0)
        for it in range(most):
            if it % 50 == 0 and bool((r.norm(dim=0) <= stop).all()):
                break
            q = self.times(values, p)
            alpha = rz / (p * q).sum(0).clamp(min=1e-300)
            x, r = x + alpha * p, r - alpha * q
            z = inv * r
            new = (r * z).sum(0)
            p, rz = z + (new / rz.clamp(min=1e-300)) * p, new
        return x

    def solve(self, currents, hc=None):
        """Newton with a backtracking line search, to the rounding of the residual."""
        cur = torch.as_tensor(currents, device=DEVICE).T
        scale = torch.ones(cur.shape[1], device=DEVICE, dtype=torch.float64) if hc is None else torch.as_tensor(hc, device=DEVICE)
        b = self.coils @ cur + self.magnet[:, None] * scale
        bn = b.norm(dim=0).clamp(min=1e-300)
        x = torch.zeros_like(b)
        last, stalled = None, 0
        for _ in range(120):
            f, values = self.system(x, True)
            r = b - f
            res = r.norm(dim=0) / bn
            worst = float(res.max())
            stalled = stalled + 1 if last is not None and worst > 0.5 * last else 0
            if worst < 3e-15 or (worst < 1e-11 and stalled >= 2):
                break
            last = worst
            d = self.cg(values, r, 1e-4)
            step = torch.ones_like(res)
            for _ in range(12):
                new = (b - self.system(x + step * d, False)[0]).norm(dim=0) / bn
                good = (new <= (1 - 1e-4 * step) * res) | (res < 1e-12)
                if bool(good.all()):
                    break
                step = torch.where(good, step, step / 2)
            x = x + step * d
        return x

    def fields(self, a):  # nodal [N, k] -> as the entry points lay them out, [k, ...]
        e = a[self.tri]
        b1, b2 = ((e * v[..., None]).sum(1) for v in self.centre)
        flux = torch.einsum("elc,elk->kc", self.coil_elements, e) * (1.0 if self.axi else self.m.depth_m)
        return [v.contiguous() for v in (a.T, b1.T, b2.T, flux)]


def exact(case, seed):
    kind = case["kind"]
    none = {"status": None, "newton": None}
    if kind == "solve":
        model, cur, hc = _solve_inputs(case, seed)
        if model.node_count * case["items"] > 2_500_000:
            return None
        f = _Fem(model)
        return dict(zip(("a", "b1", "b2", "flux"), f.fields(f.nodal(f.solve(cur, hc)))), **none)
    if kind == "meshes":
        parts = []
        for model, cur in _meshes_inputs(case, seed):
            f = _Fem(model)
            parts.append([v[0] for v in f.fields(f.nodal(f.solve(cur[None])))])
        return dict(zip(("a", "b1", "b2", "flux"), (torch.cat(v) for v in zip(*parts))), **none)
    if kind == "csr":
        model, cur = _csr_inputs(case, seed)
        b0, h0 = model.curves[0]
        nu0 = np.array(model.nu0)
        nu0[1] = h0[1] / b0[1]  # the cold operator: the secant of the table's first step
        model.curves, model.curve_index, model.nu0 = [], np.full_like(model.curve_index, -1), nu0
        f = _Fem(model)
        return {"x": f.solve(cur[None])[:, 0], "status": None}
    if kind == "tangent":
        s = prepare(case, seed)
        f = _Fem(_mesh("sector", case["size"]))
        x = torch.zeros((f.n, 1), dtype=torch.float64, device=DEVICE)
        a = torch.as_tensor(s["base"], device=DEVICE)
        on = f.row >= 0
        x[f.row[on], 0] = a[on] * f.sign[on]
        values = f.system(x, True)[1].expand(-1, case["items"]).contiguous()
        load = f.coils @ torch.as_tensor(s["directions"], device=DEVICE).T
        d = f.cg(values, load, 1e-6)
        for _ in range(3):
            d = d + f.cg(values, load - f.times(values, d), 1e-6)
        return dict(zip(("da", "db1", "db2", "dflux"), f.fields(f.nodal(d))), status=None)
    if kind == "post":
        s = prepare(case, seed)
        f = _Fem(_mesh("sector", case["size"]))
        mask = torch.as_tensor(_rotor_mask(f.m), device=DEVICE)[f.tri]
        _, _, dy, mdx = f.points[0]
        hx, hy = (mask * mdx).sum(1), -(mask * dy).sum(1)
        b1, b2 = s["fields"][1], s["fields"][2]
        w = f.area * f.m.depth_m / (2 * 4e-7 * math.pi)
        normal, shear = b1 * b1 - b2 * b2, 2 * b1 * b2
        fx, fy = w * (normal * hx + shear * hy), w * (shear * hx - normal * hy)
        return {"force": torch.stack([fx.sum(1), fy.sum(1)], 1),
                "torque": (f.cen[0] * fy - f.cen[1] * fx).sum(1), "radial_b": None, "status": None}
    x, t, p = (torch.as_tensor(v, device=DEVICE).double() for v in _network_inputs(case, seed))
    p.requires_grad_(True)
    h, o = case["hidden"], case["outputs"]
    w1, b1, w2, b2, w3, b3 = torch.split(p, [4 * h, h, h * h, h, o * h, o])
    act = torch.nn.functional.gelu
    y = act(act(x @ w1.view(h, 4).T + b1) @ w2.view(h, h).T + b2) @ w3.view(o, h).T + b3
    if case["op"] == "forward":
        return {"y": y.detach()}
    loss = 0.5 * ((y - t) ** 2).sum() / case["batch"]
    return {"loss": float(loss.detach()), "gradient": torch.autograd.grad(loss, p)[0]}
