"""Performance cases: the runs that users of the engine make, at the sizes they make them.

A case is one pass of a simulation program: hand a state to a resident model
(``set_state`` from pinned host memory), advance it, read the results back; the
contact models go on from where they are.
FP64 models return their state as doubles; mixed-precision models (FP32
element force, good to about 1e-7) are written out as single floats, as their
users store them.

``exact`` restates the same explicit step in plain torch, in 64 bits: element
by element and node by node as the textbook writes it, without the package.
"""
from __future__ import annotations

import functools
import math
import random

import numpy as np
import torch

from dynlattice_b200 import lattices
from dynlattice_b200.abi import DL_MIXED, DL_PLAIN_FP64
from dynlattice_b200.autograd import impact_objective
from dynlattice_b200.engine import Batch, Lattice

CELL = 10e-3
RADIUS = 0.5e-3
TIP_EVERY = 10
REACT_WEIGHT = -0.1
TOPOLOGIES = ("bcc", "sc", "octet")


def _rod(n_elems, steps, precision="fp64"):
    return {"kind": "rod", "elems": n_elems, "steps": steps, "precision": precision}


def _lattice(topology, n, steps, precision="mixed", plastic=True, per_strut=2, gauss=2, velocity=10.0, stepwise=False):
    return {"kind": "lattice", "topology": topology, "n": n, "steps": steps, "precision": precision,
            "plastic": plastic, "per_strut": per_strut, "gauss": gauss, "velocity": velocity, "stepwise": stepwise}


def _fibres(rods, box_mm, steps, precision="mixed"):
    return {"kind": "fibres", "rods": rods, "box_mm": box_mm, "steps": steps, "precision": precision}


def _batch(lattices_, steps, mix, n_max=12, precision="mixed"):
    return {"kind": "batch", "lattices": lattices_, "steps": steps, "mix": mix, "n_max": n_max,
            "precision": precision}


def _gradient(n, steps, precision="mixed"):
    return {"kind": "gradient", "n": n, "steps": steps, "precision": precision}


def listed():
    return [
        # one clamped rod under a ramped tip load, its tip sampled: the smallest
        # model anyone runs, thousands of steps at a time
        dict(_rod(32, 2000), name="rod32_fp64"),
        # a unit-cell study: a few cells, many short runs
        dict(_lattice("bcc", 4, 500), name="bcc4_mixed"),
        # a ragged elastic lattice in plain FP64: other topology, three elements
        # a strut, the reference's default one-point rule
        dict(_lattice("octet", 5, 300, precision="fp64", plastic=False, per_strut=3, gauss=1, velocity=5.0),
             name="octet5_elastic_fp64"),
        # elastic, mixed, one Gauss point, a size that fits no tile
        dict(_lattice("sc", 17, 300, plastic=False, gauss=1), name="sc17_elastic_mixed"),
        # the elastoplastic impact of the benchmark, in runs of 500 steps
        dict(_lattice("bcc", 20, 500), name="bcc20_mixed"),
        # the same in plain FP64, for users who want no mixed precision
        dict(_lattice("bcc", 20, 200, precision="fp64"), name="bcc20_fp64"),
        # the same driven step by step with the energies read back after each
        # (a co-simulation or a monitor in the loop)
        dict(_lattice("bcc", 20, 100, stepwise=True), name="bcc20_mixed_stepwise"),
        # a block four times as large: its working set no longer fits the L2
        dict(_lattice("bcc", 32, 100), name="bcc32_mixed"),
        # many uneven lattices stepped together (design studies)
        dict(_batch(48, 100, mix=1), name="batch48_mixed"),
        # a small fibre network in plain FP64 with rods colliding
        dict(_fibres(300, 12.331, 1000, precision="fp64"), name="fibres300_fp64"),
        # the 20 000-rod network between two plates, rods in motion
        dict(_fibres(20000, 60.0, 400), name="fibres20k_mixed"),
        # one iteration of a strut-radius optimisation: objective and gradient
        dict(_gradient(8, 800), name="gradient_bcc8_mixed"),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng: random.Random):
    kind = rng.choices(["rod", "lattice", "fibres", "batch", "gradient"], [2, 6, 2, 1, 1])[0]
    precision = rng.choice(["mixed", "mixed", "fp64"])
    if kind == "rod":
        return _rod(round(_log(rng, 4, 256)), rng.randrange(200, 2000))
    if kind == "lattice":
        topology = rng.choice(TOPOLOGIES)
        per_strut = rng.choice([1, 2, 2, 3, 4])
        plastic = rng.random() < 0.7
        gauss = 2 if plastic else rng.choice([1, 2, 3])
        per_cell = {"bcc": 8, "sc": 3, "octet": 24}[topology] * per_strut
        n = max(2, min(32, round((_log(rng, 200, 250e3) / per_cell) ** (1.0 / 3.0))))
        stepwise = rng.random() < 0.2
        elems = per_cell * n ** 3
        steps = round(_log(rng, 0.3, 1.0) * min(600.0, 30e6 / elems))
        if stepwise:
            steps = min(steps, 150)
        return _lattice(topology, n, max(20, steps), precision, plastic, per_strut, gauss,
                        round(_log(rng, 8.0, 50.0), 3), stepwise)
    if kind == "fibres":
        rods = round(_log(rng, 100, 15000))
        box = 60.0 * (rods / 20000.0) ** (1.0 / 3.0) * rng.uniform(0.9, 1.3)
        return _fibres(rods, round(box, 3), rng.randrange(100, 400), precision)
    if kind == "batch":
        return _batch(rng.randrange(2, 40), rng.randrange(40, 100), rng.randrange(1000), rng.randrange(5, 12),
                      precision)
    return _gradient(rng.randrange(3, 9), rng.randrange(100, 600), precision)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _mix(case):
    """Topology and cells of each lattice of a batch (n^3 cells, n from 4)."""
    r = random.Random(case["mix"])
    return [(r.choice(TOPOLOGIES), r.randint(4, case["n_max"])) for _ in range(case["lattices"])]


def _specs(case, seed):
    """The model (or the batch's models) and the initial velocities [N, 6]."""
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "rod":
        specs = [lattices.straight_rod(case["elems"], length=1.0 * case["elems"] / 32,
                                       tip_force=float(rng.uniform(2e3, 8e3)))]
    elif kind == "lattice":
        specs = [lattices.lattice_impact(case["topology"], n=case["n"], cell=CELL, elems_per_strut=case["per_strut"],
                                         radius=RADIUS, radius_jitter=0.05, seed=seed, velocity=case["velocity"],
                                         dt=5e-8, plastic=case["plastic"], n_gauss=case["gauss"])]
    elif kind == "gradient":
        specs = [lattices.lattice_impact("bcc", n=case["n"], cell=CELL, radius=RADIUS, seed=seed, velocity=20.0,
                                         dt=5e-8)]
    elif kind == "batch":
        specs = []
        for k, (topology, n) in enumerate(_mix(case)):
            r = float(rng.uniform(0.3e-3, 0.7e-3))
            v = float(np.exp(rng.uniform(np.log(1.0), np.log(50.0))))
            s = lattices.lattice_impact(topology, n=n, cell=CELL, radius=r, radius_jitter=0.0, seed=k, velocity=v)
            s.materials = [lattices.aluminium_elastoplastic(r)]
            s.dt = lattices.critical_dt(s)
            specs.append(s)
    else:
        specs = [lattices.fibre_network(case["rods"], box=case["box_mm"] * 1e-3, seed=seed)]
    v0 = np.concatenate([np.zeros((s.n_nodes, 6)) for s in specs])
    if kind == "fibres":
        v0[:, :3] = np.repeat(rng.normal(scale=2.0, size=(case["rods"], 3)), 5, axis=0)
    else:
        # residual motion of the free nodes, then the impacting face
        off = 0
        for s in specs:
            v = v0[off:off + s.n_nodes]
            v[:, :3] = rng.normal(scale=1e-4 if kind == "rod" else 0.01, size=(s.n_nodes, 3))
            for b in s.bcs:
                if b.kind == 0:
                    v[b.nodes, b.dof] = 0.0
            for b in s.bcs:
                if b.kind == 2:
                    v[b.nodes, b.dof] = b.factor
            off += s.n_nodes
    return specs, v0


def _pinned(a):
    t = torch.from_numpy(np.ascontiguousarray(a))
    return t.pin_memory() if torch.cuda.is_available() else t


def _precision(case):
    return DL_MIXED if case["precision"] == "mixed" else DL_PLAIN_FP64


def _out_type(case):
    return torch.float32 if case["precision"] == "mixed" else torch.float64


def prepare(case, seed):
    specs, v0 = _specs(case, seed)
    if case["kind"] == "gradient":
        radii = torch.tensor(specs[0].strut_radius, dtype=_out_type(case))
        return {"case": case, "spec": specs[0], "radii": radii}
    n = v0.shape[0]
    zeros = np.zeros((n, 3))
    state = {"case": case, "in": (_pinned(zeros), _pinned(zeros), _pinned(v0)),
             "out": (_pinned(zeros), _pinned(zeros), _pinned(np.zeros((n, 6)))), "specs": specs}
    if case["kind"] == "batch":
        state["model"] = Batch(specs, _precision(case))
    else:
        state["model"] = Lattice(specs[0], _precision(case))
    if case["kind"] == "rod":
        state["tip"] = specs[0].groups["free"]
    if case["kind"] == "fibres":
        # the plates move with the model's time, so these runs go on from where
        # they are instead of starting over
        state["model"].set_state_ptrs(*(t.data_ptr() for t in state["in"]))
    return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

_ENERGIES = ("kinetic", "potential", "dissipated", "external_work", "contact")


def _row(e, dtype):
    return torch.tensor([e[k] for k in _ENERGIES], dtype=dtype)


def run(state):
    case = state["case"]
    dtype = _out_type(case)
    if case["kind"] == "gradient":
        radii = state["radii"].detach().clone().requires_grad_(True)
        J = impact_objective(radii, state["spec"], case["steps"], react_weight=REACT_WEIGHT,
                             precision=_precision(case))
        J.backward()
        return {"objective": J.detach(), "gradient": radii.grad}
    model = state["model"]
    out = {}
    if case["kind"] == "rod":
        model.set_sampling(TIP_EVERY, state["tip"], case["steps"] // TIP_EVERY + 1)
    if case["kind"] != "fibres":
        model.set_state_ptrs(*(t.data_ptr() for t in state["in"]))
    if case.get("stepwise"):
        rows = []
        for _ in range(case["steps"]):
            model.run(1)
            rows.append(_row(model.energies(), dtype))
        out["energies"] = torch.stack(rows)
    else:
        model.run(case["steps"])
        if case["kind"] == "batch":
            out["energies"] = torch.stack([_row(model.lattice_energies(k), dtype) for k in range(case["lattices"])])
        else:
            out["energies"] = _row(model.energies(), dtype)
    if case["kind"] == "rod":
        steps, rows, energies = model.samples()
        out["sample_steps"], out["sample_rows"] = steps, torch.from_numpy(rows).to(dtype)
        out["sample_energies"] = torch.from_numpy(energies).to(dtype)
    if case["kind"] == "fibres":
        out["plates"] = torch.from_numpy(model.plate_reaction()).to(dtype)
    model.get_state_ptrs(*(t.data_ptr() for t in state["out"]))
    out["u"], out["theta"], out["v"] = (t.to(dtype) for t in state["out"])
    return out


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

@functools.lru_cache(maxsize=None)
def _count(topology, n, per_strut):
    struts = lattices.lattice_struts(topology, n, CELL)
    return struts[1].shape[0] * per_strut, struts[0].shape[0] + struts[1].shape[0] * (per_strut - 1)


def _sizes(case):
    """Elements, nodes, Gauss points per element, whether plastic."""
    kind = case["kind"]
    if kind == "rod":
        return case["elems"], case["elems"] + 1, 2, False
    if kind == "lattice":
        return (*_count(case["topology"], case["n"], case["per_strut"]), case["gauss"], case["plastic"])
    if kind == "gradient":
        return (*_count("bcc", case["n"], 2), 2, True)
    if kind == "fibres":
        return 4 * case["rods"], 5 * case["rods"], 1, False
    counts = [_count(t, n, 2) for t, n in _mix(case)]
    return sum(c[0] for c in counts), sum(c[1] for c in counts), 2, True


def work(case):
    """Bytes: state in and out (12 values a node each way), the constants of
    nodes and elements and the plastic history (both ways), once a pass.
    Operations: what one element, Gauss point, return-map check and node take
    in one step."""
    E, N, G, plastic = _sizes(case)
    real = 4 if case["precision"] == "mixed" else 8
    out = 4 if case["precision"] == "mixed" else 8
    node = 12 * 8 + 12 * out + 8 + 7 * real
    elem = 8 + 8 + 8 * real + 6 * real + (G * 2 * 15 * real if plastic else 0)
    flops = (220 + G * (190 + (60 if plastic else 0))) * E + 330 * N
    reverse = 3 if case["kind"] == "gradient" else 1
    return {"bytes": float(N * node + E * elem), "flops": float(flops) * case["steps"] * reverse}


# ---------------------------------------------------------------------------
# the same in 64 bits, in plain torch
# ---------------------------------------------------------------------------

_GAUSS = {1: ([0.0], [2.0]), 2: ([-1 / math.sqrt(3.0), 1 / math.sqrt(3.0)], [1.0, 1.0]),
          3: ([-math.sqrt(0.6), 0.0, math.sqrt(0.6)], [5.0 / 9.0, 8.0 / 9.0, 5.0 / 9.0])}


def _qmul(a, b):
    aw, av, bw, bv = a[..., :1], a[..., 1:], b[..., :1], b[..., 1:]
    w = aw * bw - (av * bv).sum(-1, keepdim=True)
    return torch.cat([w, aw * bv + bw * av + torch.linalg.cross(av, bv)], -1)


def _qconj(q):
    return torch.cat([q[..., :1], -q[..., 1:]], -1)


def _qrot(q, v):
    t = 2.0 * torch.linalg.cross(q[..., 1:], v)
    return v + q[..., :1] * t + torch.linalg.cross(q[..., 1:], t)


def _sinc(x2):
    """sin(x)/x of x^2, differentiable at 0."""
    small = x2 < 1e-4
    x = torch.sqrt(torch.where(small, torch.ones_like(x2), x2))
    return torch.where(small, 1 - x2 / 6 + x2 * x2 / 120 - x2 ** 3 / 5040, torch.sin(x) / x)


def _qexp(phi):
    t2 = 0.25 * (phi * phi).sum(-1, keepdim=True)
    small = t2 < 1e-4
    t = torch.sqrt(torch.where(small, torch.ones_like(t2), t2))
    w = torch.where(small, 1 - t2 / 2 + t2 * t2 / 24 - t2 ** 3 / 720, torch.cos(t))
    return torch.cat([w, 0.5 * _sinc(t2) * phi], -1)


def _qlog(q):
    q = torch.where(q[..., :1] < 0, -q, q)
    w, u = q[..., :1], q[..., 1:]
    s2 = (u * u).sum(-1, keepdim=True)
    r = s2 / (w * w)
    small = r < 1e-4
    s = torch.sqrt(torch.where(small, torch.ones_like(s2), s2))
    f = torch.where(small, 2 / w * (1 - r / 3 + r * r / 5 - r ** 3 / 7 + r ** 4 / 9), 2 * torch.atan2(s, w) / s)
    return f * u


def _qhalf(q):
    q = torch.where(q[..., :1] < 0, -q, q)
    h = torch.cat([q[..., :1] + 1.0, q[..., 1:]], -1)
    return h / torch.linalg.vector_norm(h, dim=-1, keepdim=True)


def _qmat(q):
    w, x, y, z = q.unbind(-1)
    return torch.stack([w * w + x * x - y * y - z * z, 2 * (x * y - w * z), 2 * (x * z + w * y),
                        2 * (x * y + w * z), w * w - x * x + y * y - z * z, 2 * (y * z - w * x),
                        2 * (x * z - w * y), 2 * (y * z + w * x), w * w - x * x - y * y + z * z],
                       -1).reshape(*q.shape[:-1], 3, 3)


class _Exact:
    """One model, or the union of a batch, with the explicit step of it."""

    def __init__(self, specs, device):
        self.dev = device
        t = functools.partial(torch.as_tensor, device=device)
        node_off = np.cumsum([0] + [s.n_nodes for s in specs])
        self.X0 = t(np.concatenate([s.coords for s in specs]))
        self.conn = t(np.concatenate([s.conn.astype(np.int64) + o for s, o in zip(specs, node_off)]))
        N = self.N = self.X0.shape[0]
        self.E = self.conn.shape[0]
        self.G = specs[0].n_gauss
        per_node = lambda vals: t(np.concatenate([np.full(s.n_nodes, x) for s, x in zip(specs, vals)]))
        per_elem = lambda f: t(np.concatenate([np.broadcast_to(f(s), (s.n_elems,)) for s in specs]).copy())
        self.dt = per_node([s.dt for s in specs])[:, None]
        self.lattice_of_node = per_node(range(len(specs))).long()
        self.lattice_of_elem = self.lattice_of_node[self.conn[:, 0]]
        self.n_lattices = len(specs)
        m = specs[0].materials[0]
        self.mat, self.plastic = m, m.yield_cond is not None
        self.young, self.shear, self.ks, self.rho = m.young, m.shear_modulus, m.shear_correction, m.density
        self.H = m.isotropic_coefficient or 0.0
        self.prec, self.max_iter = m.precision, m.max_iter
        self.sy = lattices.SIGMA_Y_AL
        chord = self.X0[self.conn[:, 1]] - self.X0[self.conn[:, 0]]
        self.L0 = torch.linalg.vector_norm(chord, dim=1)
        tan = chord / self.L0[:, None]
        c = tan[:, 2]
        flip = c < -1 + 1e-12
        q = torch.stack([1 + c, -tan[:, 1], tan[:, 0], torch.zeros_like(c)], 1)
        q = torch.where(flip[:, None], t([0.0, 1.0, 0.0, 0.0]).double(), q)
        self.frame = q / torch.linalg.vector_norm(q, dim=1, keepdim=True)
        self.set_radius(per_elem(lambda s: s.elem_radius if s.elem_radius is not None else s.materials[0].radius))
        # loads and constraints: a constrained DOF keeps its velocity
        self.free = torch.ones(N, 6, dtype=torch.float64, device=device)
        self.load = torch.zeros(N, 6, dtype=torch.float64, device=device)
        self.ramp = 0
        for s, o in zip(specs, node_off):
            for b in s.bcs:
                idx = t(b.nodes.astype(np.int64) + int(o))
                if b.kind == 0:
                    self.free[idx, b.dof] = 0.0
                elif b.kind == 1:
                    self.load[idx, b.dof] += b.factor
                    self.ramp = 500
        self.contact = specs[0].contact
        self.elem_rod = t(np.concatenate([s.elem_rod.astype(np.int64) for s in specs]))
        self.top = t(specs[0].groups["top"].astype(np.int64)) if "top" in specs[0].groups else None

    def set_radius(self, r):
        A, I = math.pi * r ** 2, math.pi * r ** 4 / 4
        J = 2 * I
        gka, ea = self.shear * self.ks * A, self.young * A
        self.C = torch.stack([gka, gka, ea, self.young * I, self.young * I, self.shear * J], 1)
        self.r, self.A = r, A
        L, rho = self.L0, self.rho
        d = torch.stack([rho * I * L + rho * A * L ** 3 / 12] * 2 + [rho * J * L], 1)
        F = _qmat(self.frame)
        S = 0.5 * (F * d[:, None, :]) @ F.transpose(1, 2)
        half = 0.5 * rho * A * L
        zero = torch.zeros(self.N, dtype=torch.float64, device=self.dev)
        zero3 = torch.zeros(self.N, 3, 3, dtype=torch.float64, device=self.dev)
        i, j = self.conn[:, 0], self.conn[:, 1]
        self.mass = zero.index_add(0, i, half).index_add(0, j, half)
        self.S = zero3.index_add(0, i, S).index_add(0, j, S)
        self.Sinv = torch.linalg.inv(self.S)
        sy = self.sy
        n_p, v_p = sy * A, sy / math.sqrt(3.0) * A
        m_p, t_p = sy * 4.0 / 3.0 * r ** 3, sy / math.sqrt(3.0) * 2.0 / 3.0 * math.pi * r ** 3
        self.cap = torch.stack([v_p, v_p, n_p, m_p, m_p, t_p], 1)
        self.dfdh = 1.0 / (sy * torch.sqrt(A))

    def start(self, v0):
        z = functools.partial(torch.zeros, dtype=torch.float64, device=self.dev)
        rot = z(self.N, 4)
        rot[:, 0] = 1.0
        E, G = (self.E, self.G) if self.plastic else (0, 0)
        return (self.X0.clone(), rot, torch.as_tensor(v0, device=self.dev).clone(), z(E, G, 6), z(E, G), z(E, G, 6),
                z(E, G))

    def _material(self, eps, g, C, hist):
        """Stress of Gauss point g, its history after the step (return map by
        cutting planes) and the strains' elastic part."""
        if not self.plastic:
            return C * eps, None, eps
        ep0, al0, old, ed = (h[:, g] for h in hist)
        ep, al = ep0, al0
        todo = torch.arange(self.E, device=self.dev)
        for _ in range(self.max_iter):
            Cs, cap, dh = C[todo], self.cap[todo], self.dfdh[todo]
            sig = Cs * (eps[todo] - ep[todo])
            s2 = ((sig / cap) ** 2).sum(1)
            keep = torch.sqrt(s2.detach()) - 1 - self.H * al[todo].detach() * dh.detach() >= self.prec
            todo, Cs, cap, dh, sig, s2 = todo[keep], Cs[keep], cap[keep], dh[keep], sig[keep], s2[keep]
            if todo.numel() == 0:
                break
            s = torch.sqrt(s2)
            f = s - 1 - self.H * al[todo] * dh
            gr = sig / cap ** 2 / s[:, None]
            flow = f / ((gr * gr * Cs).sum(1) + self.H * dh * dh)
            ep = ep.index_add(0, todo, flow[:, None] * gr)
            al = al.index_add(0, todo, flow * dh)
        sig = C * (eps - ep)
        ed = ed + ((C * (old - ep0) + sig) / 2 * (ep - ep0)).sum(1)
        return sig, (ep, al, eps, ed), eps - ep

    def element_force(self, state):
        """End forces added up per node [N, 6], the history after the step,
        stored and dissipated energy per element."""
        x, rot, _, *hist = state
        i, j = self.conn[:, 0], self.conn[:, 1]
        Li, Lj = _qmul(rot[i], self.frame), _qmul(rot[j], self.frame)
        rel = _qmul(_qconj(Li), Lj)
        phi = _qlog(rel)
        ref = _qmul(Li, _qhalf(rel))
        dx = (x[j] - x[i]) / self.L0[:, None]
        e3 = torch.tensor([0.0, 0.0, 1.0], dtype=torch.float64, device=self.dev)
        fi = torch.zeros(self.E, 6, dtype=torch.float64, device=self.dev)
        fj = torch.zeros_like(fi)
        pot = torch.zeros(self.E, dtype=torch.float64, device=self.dev)
        diss = torch.zeros_like(pot)
        new = []
        for g, (xi, W) in enumerate(zip(*_GAUSS[self.G])):
            L = _qmul(ref, _qexp(0.5 * xi * phi))
            eps = torch.cat([_qrot(_qconj(L), dx) - e3, phi / self.L0[:, None]], 1)
            sig, h, el = self._material(eps, g, self.C, hist)
            n, m = _qrot(L, sig[:, :3]), _qrot(L, sig[:, 3:])
            w = (0.5 * W * self.L0)[:, None]
            pxn = torch.linalg.cross(dx, n)
            ni, nj = 0.5 * (1 - xi), 0.5 * (1 + xi)
            fi = fi + torch.cat([-0.5 * W * n, -0.5 * W * m - w * ni * pxn], 1)
            fj = fj + torch.cat([0.5 * W * n, 0.5 * W * m - w * nj * pxn], 1)
            pot = pot + 0.5 * w[:, 0] * (el * sig).sum(1)
            if h is not None:
                new.append(h)
                diss = diss + w[:, 0] * h[3]
        hist = tuple(torch.stack([h[k] for h in new], 1) for k in range(4)) if new else tuple(hist)
        f = torch.zeros(self.N, 6, dtype=torch.float64, device=self.dev)
        return f.index_add(0, i, fi).index_add(0, j, fj), hist, pot, diss

    def advance(self, state, f, hist, step, fields=None):
        """Node update: block mass solve, v += dt a, x += dt v, R = exp(dt w) R."""
        x, rot, v = state[:3]
        load = self.load * min(step / self.ramp, 1.0) if self.ramp else None
        r = -f if load is None else load - f
        R = _qmat(rot)
        body = lambda a: (R.transpose(1, 2) @ a[:, :, None])[:, :, 0]
        space = lambda a: (R @ a[:, :, None])[:, :, 0]
        w = body(v[:, 3:])
        Mw = (self.S @ w[:, :, None])[:, :, 0]
        mom = body(r[:, 3:]) - torch.linalg.cross(w, Mw)
        acc = torch.cat([r[:, :3] / self.mass[:, None], space((self.Sinv @ mom[:, :, None])[:, :, 0])], 1)
        v = v + self.dt * (self.free * acc)
        x = x + self.dt * v[:, :3]
        new = _qmul(_qexp(self.dt * v[:, 3:]), rot)
        new = new / torch.linalg.vector_norm(new, dim=1, keepdim=True)
        if fields is not None:
            w1 = body(v[:, 3:])
            fields["kinetic"] = 0.5 * (self.mass * (v[:, :3] ** 2).sum(1) + (w1 * (self.S @ w1[:, :, None])[:, :, 0]).sum(1))
            if load is not None:
                fields["work"] = (load * self.dt * v).sum()
        return (x, new, v, *hist)

    # -- rod--rod contact and plates -----------------------------------------

    def find_pairs(self, reach):
        """Element pairs of different rods whose segments may come within 2r
        while no node moves more than `reach`."""
        x = self.X0
        a, b = x[self.conn[:, 0]], x[self.conn[:, 1]]
        mid, half = 0.5 * (a + b), 0.5 * self.L0.max()
        far = 2 * half + 2 * self.contact.radius + 2 * reach
        order = torch.argsort(mid[:, 2])
        zs = mid[order, 2].contiguous()
        found = []
        for at in range(0, self.E, 2048):
            rows = order[at:at + 2048]
            hi = int(torch.searchsorted(zs, zs[min(at + 2048, self.E) - 1] + far))
            cols = order[at:hi]
            near = torch.cdist(mid[rows], mid[cols]) <= far
            p, q = near.nonzero(as_tuple=True)
            ok = (p < q) & (self.elem_rod[rows[p]] != self.elem_rod[cols[q]])
            found.append(torch.stack([rows[p[ok]], cols[q[ok]]], 1))
        pairs = torch.cat(found)
        swap = self.elem_rod[pairs[:, 0]] > self.elem_rod[pairs[:, 1]]
        pairs = torch.where(swap[:, None], pairs.flip(1), pairs)
        nodes = torch.cat([self.conn[pairs[:, 0]], self.conn[pairs[:, 1]]], 1)
        keep = self._segment_gap(x, nodes) <= 2 * self.contact.radius + 2 * reach
        self.pair_nodes = nodes[keep]

    @staticmethod
    def _segment_gap(x, nodes):
        """Distance of two segments (clamped closest points)."""
        p, q = x[nodes[:, 0]], x[nodes[:, 2]]
        d1, d2, r = x[nodes[:, 1]] - p, x[nodes[:, 3]] - q, p - q
        a, e, f = (d1 * d1).sum(1), (d2 * d2).sum(1), (d2 * r).sum(1)
        c, b = (d1 * r).sum(1), (d1 * d2).sum(1)
        den = a * e - b * b
        s = torch.where(den > 1e-300, ((b * f - c * e) / den).clamp(0, 1), torch.zeros_like(a))
        t = (b * s + f) / e
        s = torch.where(t < 0, (-c / a).clamp(0, 1), torch.where(t > 1, ((b - c) / a).clamp(0, 1), s))
        t = t.clamp(0, 1)
        return torch.linalg.vector_norm(p + s[:, None] * d1 - q - t[:, None] * d2, dim=1)

    def contact_force(self, x, t):
        """Penalty forces of closed pairs and plates [N, 3], their energy, the plates' reactions."""
        r, k = self.contact.radius, self.contact.penalty
        f = torch.zeros(self.N, 3, dtype=torch.float64, device=self.dev)
        energy = torch.zeros((), dtype=torch.float64, device=self.dev)
        nodes = self.pair_nodes
        if nodes.shape[0]:
            nodes = nodes[self._segment_gap(x, nodes) <= 2 * r * (1 + 1e-6)]
        if nodes.shape[0]:
            A, B = (x[nodes[:, 0]], x[nodes[:, 1]]), (x[nodes[:, 2]], x[nodes[:, 3]])
            tA, tB = A[1] - A[0], B[1] - B[0]
            d = B[1] + B[0] - A[1] - A[0]
            dot = lambda a, b: (a * b).sum(1)
            aa, bb, ab = dot(tA, tA), dot(tB, tB), dot(tA, tB)
            den = bb * aa - ab * ab
            uA = -dot(d, tB * ab[:, None] - tA * bb[:, None]) / den
            uB = dot(d, tA * ab[:, None] - tB * aa[:, None]) / den
            inside = lambda u: (u >= -1) & (u <= 1)
            project = lambda s, M: (2 * dot(s, M[1] - M[0]) - dot(M[1] - M[0], M[1] + M[0])) / dot(M[1] - M[0], M[1] - M[0])
            point = lambda M, u: (0.5 * (1 - u))[:, None] * M[0] + (0.5 * (1 + u))[:, None] * M[1]

            def push(on, weights, gap_vec):
                """Pairs `on`: force k gap n on their four nodes with the given weights."""
                nonlocal f, energy
                dist = torch.linalg.vector_norm(gap_vec, dim=1)
                on = on & (dist > 0) & (dist <= 2 * r)
                if not bool(on.any()):
                    return
                gap = dist[on] - 2 * r
                s = k * gap[:, None] * gap_vec[on] / dist[on][:, None]
                for c in range(4):
                    f = f.index_add(0, nodes[on, c], weights[c][on][:, None] * s)
                energy = energy + 0.5 * k * (gap * gap).sum()

            zero, one = torch.zeros_like(uA), torch.ones_like(uA)
            ends = lambda u: (0.5 * (1 - u), 0.5 * (1 + u))
            inA, inB = inside(uA), inside(uB)
            a0, a1 = ends(uA)
            b0, b1 = ends(uB)
            push(inA & inB, (-a0, -a1, b0, b1), point(B, uB) - point(A, uA))
            for end in (0, 1):
                isA = (uA < -1) if end == 0 else ~(uA < -1)
                # one-sided: the node of A against B, at the abscissa of B's node on A
                u = project(B[end], A)
                m0, m1 = ends(u)
                ws = [zero, zero, m0, m1]
                ws[end] = -one
                push(~inA & inB & isA & inside(u), ws, point(B, u) - A[end])
                isB = (uB < -1) if end == 0 else ~(uB < -1)
                u = project(B[end], A)
                m0, m1 = ends(u)
                ws = [m0, m1, zero, zero]
                ws[2 + end] = -one
                push(inA & ~inB & isB & inside(u), ws, point(A, u) - B[end])
                # both outside: every end against the other segment
                u = project(A[end], B)
                m0, m1 = ends(u)
                ws = [zero, zero, m0, m1]
                ws[end] = -one
                push(~inA & ~inB & inside(u), ws, point(B, u) - A[end])
                u = project(B[end], A)
                m0, m1 = ends(u)
                ws = [m0, m1, zero, zero]
                ws[2 + end] = -one
                push(~inA & ~inB & inside(u), ws, point(A, u) - B[end])
        plates = torch.zeros(2, 3, dtype=torch.float64, device=self.dev)
        for p, plate in enumerate(self.contact.plates):
            n = torch.tensor(plate["normal"], dtype=torch.float64, device=self.dev)
            at = torch.tensor(plate["point0"], dtype=torch.float64, device=self.dev) + t * torch.tensor(
                plate["velocity"], dtype=torch.float64, device=self.dev)
            gap = torch.clamp((x - at) @ n - r, max=0.0)
            kg = plate["penalty"] * gap
            f = f + kg[:, None] * n
            plates[p] = kg.sum() * n
            energy = energy + 0.5 * (kg * gap).sum()
        return f, energy, plates

    def step(self, state, step, t=0.0, fields=None):
        f, hist, pot, diss = self.element_force(state)
        if fields is not None:
            fields["potential"], fields["dissipated"] = pot, diss
        if self.contact is not None:
            fc, energy, plates = self.contact_force(state[0], t)
            f = torch.cat([f[:, :3] + fc, f[:, 3:]], 1)
            if fields is not None:
                fields["contact"], fields["plates"] = energy, plates
        if fields is not None and self.top is not None:
            fields["reaction"] = f[self.top, 2].sum()
        return self.advance(state, f, hist, step, fields)


def _per_lattice(model, fields):
    z = torch.zeros(model.n_lattices, 5, dtype=torch.float64, device=model.dev)
    z[:, 0] = z[:, 0].index_add(0, model.lattice_of_node, fields["kinetic"])
    z[:, 1] = z[:, 1].index_add(0, model.lattice_of_elem, fields["potential"])
    z[:, 2] = z[:, 2].index_add(0, model.lattice_of_elem, fields["dissipated"])
    return z


def _exact_gradient(model, spec, case, v0, radii):
    """Objective and its gradient: the step differentiated by torch, segment by segment."""
    steps, seg = case["steps"], 10
    rod = torch.as_tensor(spec.elem_rod.astype(np.int64), device=model.dev)
    r = radii.to(model.dev, torch.float64).requires_grad_(True)
    with torch.no_grad():
        model.set_radius(r[rod])
        state, saved, peak, at = model.start(v0), [], 0.0, 1
        for k in range(1, steps + 1):
            if (k - 1) % seg == 0:
                saved.append(state)
            fields = {}
            state = model.step(state, k, fields=fields)
            if abs(float(fields["reaction"])) > abs(peak):
                peak, at = float(fields["reaction"]), k
        diss = float(fields["dissipated"].sum())
    sign = -1.0 if peak < 0 else 1.0
    w = torch.stack([0.5 * W * model.L0 for W in _GAUSS[model.G][1]], 1)
    back = [torch.zeros_like(s) for s in state[:-1]] + [w]
    grad = torch.zeros_like(r)
    for c in range(len(saved) - 1, -1, -1):
        first = [s.detach().requires_grad_(True) for s in saved[c]]
        saved[c] = None
        with torch.enable_grad():
            model.set_radius(r[rod])
            state, extra = tuple(first), 0.0
            for k in range(c * seg + 1, min(steps, (c + 1) * seg) + 1):
                fields = {}
                state = model.step(state, k, fields=fields)
                if k == at:
                    extra = REACT_WEIGHT * sign * fields["reaction"]
            total = sum((s * b).sum() for s, b in zip(state, back)) + extra
        got = torch.autograd.grad(total, first + [r], allow_unused=True)
        back = [torch.zeros_like(s) if b is None else b for s, b in zip(first, got)]
        grad = grad + got[-1]
        model.set_radius(r.detach()[rod])
    return {"objective": torch.tensor(diss + REACT_WEIGHT * abs(peak), dtype=torch.float64), "gradient": grad.detach()}


def exact(case, seed):
    device = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    specs, v0 = _specs(case, seed)
    model = _Exact(specs, device)
    if case["kind"] == "gradient":
        return _exact_gradient(model, specs[0], case, _impact_velocity(specs[0]),
                               torch.tensor(specs[0].strut_radius, dtype=_out_type(case)))
    with torch.no_grad():
        if model.contact is not None:
            fastest = float(np.linalg.norm(v0[:, :3], axis=1).max()) + 5.0
            model.find_pairs(1.5 * fastest * specs[0].dt * case["steps"])
        state = model.start(v0)
        work_done, per_step, sampled, rows = 0.0, [], [], []
        for k in range(1, case["steps"] + 1):
            last = k == case["steps"]
            sample = case["kind"] == "rod" and k % TIP_EVERY == 0
            fields = {} if (last or sample or case.get("stepwise") or model.ramp) else None
            state = model.step(state, k, t=k * specs[0].dt, fields=fields)
            if fields is None:
                continue
            work_done = work_done + fields.get("work", 0.0)
            z = _per_lattice(model, fields)
            if case["kind"] != "batch":
                z[0, 3] = work_done
                z[0, 4] = fields.get("contact", 0.0)
            if sample:
                tip = int(specs[0].groups["free"][0])
                rows.append(torch.cat([state[0][tip] - model.X0[tip], _qlog(state[1][tip]), state[2][tip]]))
                sampled.append(z[0].clone())
            if last or case.get("stepwise"):
                per_step.append(z)
        out = {}
        if case.get("stepwise"):
            out["energies"] = torch.cat(per_step)
        else:
            out["energies"] = per_step[-1] if case["kind"] == "batch" else per_step[-1][0]
        if case["kind"] == "rod":
            out["sample_steps"] = torch.arange(TIP_EVERY, case["steps"] + 1, TIP_EVERY)
            out["sample_rows"], out["sample_energies"] = torch.stack(rows)[:, None, :], torch.stack(sampled)
        if case["kind"] == "fibres":
            out["plates"] = fields["plates"]
        out["u"], out["theta"], out["v"] = state[0] - model.X0, _qlog(state[1]), state[2]
        return out


def _impact_velocity(spec):
    """The objective's own start: at rest, the impacting face in motion."""
    v = np.zeros((spec.n_nodes, 6))
    for b in spec.bcs:
        if b.kind == 2:
            v[b.nodes, b.dof] = b.factor
    return v
