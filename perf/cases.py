"""Timed cases of the SIMP hot path, through the package's public entry points.

``listed()`` holds the sizes that the package is used at: the reference's small
cantilever, odd grids of a batch of designs, the 128x64x64 workload of the
throughput benchmark in both precisions, the 256x128x128 design, the
differentiation workload and the single layers (density filter and projection
with its chain rule, OC update, linear solve).  ``draw(rng)`` gives one more case
of the same ranges.  ``prepare`` builds what a program holds before the call,
``run`` is one pass, ``exact`` restates a pass in plain 64-bit torch.
"""

from __future__ import annotations

import itertools
import math

import numpy as np
import torch

ETA, MOVE, PENAL = 0.5, 0.2, 3.0
EMIN = 1.0e-9
# corner offsets (x, y, z) of the hexahedron in its local order
CORNERS = ((0, 0, 0), (0, 1, 0), (1, 1, 0), (1, 0, 0), (0, 0, 1), (0, 1, 1), (1, 1, 1), (1, 0, 1))


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _loop(name, nelx, nely, nelz, precision, volfrac, rmin, beta, masks, steps=3):
    return {"name": name, "kind": "loop", "nelx": nelx, "nely": nely, "nelz": nelz, "precision": precision,
            "volfrac": volfrac, "rmin": rmin, "beta": beta, "masks": masks, "steps": steps}


def listed():
    return [
        # a whole optimization call as a script makes it: host arrays in and out, default
        # options (FP64), two projection stages on the reference's small cantilever
        {"name": "top3d_32x16x16", "kind": "top3d", "nelx": 32, "nely": 16, "nelz": 16, "volfrac": 0.3,
         "rmin": 3.0, "maxloop": 3},
        # loop bodies of a run that continues from a design (the first solve starts cold, the
        # next ones from the last solutions): the small grid, where launches and latency count
        _loop("loop_fp64_32x16x16", 32, 16, 16, "fp64", 0.3, 3.0, 1.0, False),
        # an odd grid of the kind a batch of designs holds, with a steeper projection
        _loop("loop_mixed_61x30x37", 61, 30, 37, "mixed", 0.25, 2.3, 4.0, True),
        # the throughput benchmark's workload in its two precisions
        _loop("loop_mixed_128x64x64", 128, 64, 64, "mixed", 0.3, 3.0, 1.0, True),
        _loop("loop_fp64_128x64x64", 128, 64, 64, "fp64", 0.3, 3.0, 1.0, True),
        # the largest single design that the benchmark runs
        _loop("loop_mixed_256x128x128", 256, 128, 128, "mixed", 0.2, 4.5, 2.0, True),
        # compliance of a design as an autograd function: forward and backward, three load
        # cases, displacements recomputed in backward (the default)
        {"name": "gradient_48x24x24", "kind": "gradient", "nelx": 48, "nely": 24, "nelz": 24, "rmin": 2.5,
         "beta": 4.0, "recompute": True},
        # independent designs of uneven sizes advanced by one graph launch
        {"name": "batch_12", "kind": "batch", "designs": 12, "spec_seed": 0, "steps": 2},
        # density filter, projection and the chain rule back through them
        {"name": "density_128x64x64", "kind": "density", "nelx": 128, "nely": 64, "nelz": 64, "rmin": 3.0,
         "beta": 2.0},
        # the same at the smallest sizes: latency of the call
        {"name": "density_24x12x13", "kind": "density", "nelx": 24, "nely": 12, "nelz": 13, "rmin": 1.5,
         "beta": 8.0},
        # the optimality-criteria update alone
        {"name": "oc_96x48x45", "kind": "oc", "nelx": 96, "nely": 48, "nelz": 45, "rmin": 2.5, "beta": 4.0,
         "volfrac": 0.35},
        # one linear solve from zero with a new density, for programs with a loop of their own
        {"name": "solve_mixed_107x53x45", "kind": "solve", "nelx": 107, "nely": 53, "nelz": 45,
         "precision": "mixed", "volfrac": 0.4},
    ]


def _draw_grid(rng, lo, hi):
    """A grid of lo to hi elements (log-uniform), roughly 2:1:1 with odd sizes among them."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    a = (n / 2.0) ** (1.0 / 3.0)
    nelx = int(round(2 * a * rng.uniform(0.8, 1.25)))
    nely = int(round(a * rng.uniform(0.8, 1.25)))
    nelz = max(8, int(n / (nelx * nely)))
    return max(12, nelx), max(8, nely), nelz


def draw(rng):
    kind = rng.choice(["loop", "loop", "loop", "solve", "density", "density", "oc", "gradient", "top3d", "batch"])
    if kind == "loop":
        precision = rng.choice(["mixed", "mixed", "fp64"])
        nelx, nely, nelz = _draw_grid(rng, 5.0e3, 1.5e6 if precision == "mixed" else 4.0e5)
        c = _loop("", nelx, nely, nelz, precision, round(rng.uniform(0.15, 0.4), 3), round(rng.uniform(1.5, 4.5), 2),
                  rng.choice([1.0, 2.0, 4.0]), rng.random() < 0.7)
        del c["name"]
        return c
    if kind == "solve":
        precision = rng.choice(["mixed", "fp64"])
        nelx, nely, nelz = _draw_grid(rng, 5.0e3, 1.0e6 if precision == "mixed" else 4.0e5)
        return {"kind": kind, "nelx": nelx, "nely": nely, "nelz": nelz, "precision": precision,
                "volfrac": round(rng.uniform(0.2, 0.5), 3)}
    if kind == "density":
        nelx, nely, nelz = _draw_grid(rng, 2.0e3, 4.0e6)
        return {"kind": kind, "nelx": nelx, "nely": nely, "nelz": nelz, "rmin": round(rng.uniform(1.3, 6.0), 2),
                "beta": rng.choice([1.0, 2.0, 4.0, 8.0])}
    if kind == "oc":
        nelx, nely, nelz = _draw_grid(rng, 2.0e3, 2.0e6)
        return {"kind": kind, "nelx": nelx, "nely": nely, "nelz": nelz, "rmin": round(rng.uniform(1.3, 4.5), 2),
                "beta": rng.choice([1.0, 2.0, 4.0, 8.0]), "volfrac": round(rng.uniform(0.2, 0.5), 3)}
    if kind == "gradient":
        nelx, nely, nelz = _draw_grid(rng, 4.0e3, 1.5e5)
        return {"kind": kind, "nelx": nelx, "nely": nely, "nelz": nelz, "rmin": round(rng.uniform(1.5, 3.5), 2),
                "beta": rng.choice([1.0, 2.0, 4.0]), "recompute": rng.random() < 0.5}
    if kind == "top3d":
        nelx, nely, nelz = _draw_grid(rng, 3.0e3, 4.0e4)
        return {"kind": kind, "nelx": nelx, "nely": nely, "nelz": nelz, "volfrac": round(rng.uniform(0.25, 0.45), 3),
                "rmin": round(rng.uniform(1.5, 3.0), 2), "maxloop": rng.randint(2, 4)}
    return {"kind": kind, "designs": rng.randint(4, 12), "spec_seed": rng.randint(1, 10 ** 6), "steps": 2}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _field(shape, seed, waves=12):
    """Smooth seeded random field of unit variance on the grid (cosine waves of a few
    elements to the whole length), on the GPU: the structure of a design in progress."""
    rng = np.random.default_rng(seed)
    nely, nelx, nelz = shape
    y = torch.arange(nely, dtype=torch.float64, device="cuda")[:, None, None]
    x = torch.arange(nelx, dtype=torch.float64, device="cuda")[None, :, None]
    z = torch.arange(nelz, dtype=torch.float64, device="cuda")[None, None, :]
    out = torch.zeros(shape, dtype=torch.float64, device="cuda")
    for _ in range(waves):
        k = rng.normal(size=3)
        k *= 2.0 * math.pi / (math.exp(rng.uniform(math.log(8.0), math.log(64.0))) * np.linalg.norm(k))
        out += torch.cos(k[0] * x + k[1] * y + k[2] * z + rng.uniform(0.0, 2.0 * math.pi))
    return out * math.sqrt(2.0 / waves)


def _fortran(t):
    """The same (nely, nelx, nelz) values in the package's element order (y fastest)."""
    return t.permute(2, 1, 0).contiguous().permute(2, 1, 0)


def _shape(c):
    return c["nely"], c["nelx"], c["nelz"]


def _masks(c):
    """Protected solid and void masks: the load strip and the clamped face, and with
    ``masks`` a void cylinder along y and a solid slab at the clamped end."""
    nely, nelx, nelz = shape = _shape(c)
    solid, void = np.zeros(shape, bool), np.zeros(shape, bool)
    if c.get("masks"):
        r = max(2, 12 * nelx // 128)
        _, xx, zz = np.ogrid[:nely, :nelx, :nelz]
        void |= (xx - nelx // 2) ** 2 + (zz - nelz // 2) ** 2 <= r * r
        solid[:, : max(1, 4 * nelx // 128), :] = True
    solid[:, -1, 0] = True
    solid[:, 0, :] = True
    solid &= ~void
    return solid, void


def _design(c, seed, solid=None, void=None):
    """A design in progress: volfrac on average, smooth variation, protected elements set."""
    x = (c["volfrac"] * (1.0 + 0.7 * _field(_shape(c), seed))).clamp(0.02, 1.0)
    if solid is not None:
        x[torch.as_tensor(solid, device="cuda")] = 1.0
        x[torch.as_tensor(void, device="cuda")] = 0.0
    return _fortran(x)


def _node(c, ix, iy, iz):
    return iy + (c["nely"] + 1) * (ix + (c["nelx"] + 1) * iz)


def _edge_load(c, comp=2, iz=0):
    """Total unit load along the x = nelx edge at height iz, in direction comp."""
    F = np.zeros(3 * (c["nelx"] + 1) * (c["nely"] + 1) * (c["nelz"] + 1))
    for iy in range(c["nely"] + 1):
        F[3 * _node(c, c["nelx"], iy, iz) + comp] = (-1.0 if comp == 2 else 1.0) / (c["nely"] + 1)
    return F


def _load_cases(c):
    Fp = np.zeros(3 * (c["nelx"] + 1) * (c["nely"] + 1) * (c["nelz"] + 1))
    Fp[3 * _node(c, c["nelx"], c["nely"] // 2, c["nelz"] // 2) + 2] = -1.0
    return np.stack([_edge_load(c), _edge_load(c, 1, c["nelz"]), Fp])


def _fixed(c):
    """All DOFs of the face x = 0."""
    m = np.zeros((c["nelz"] + 1, c["nelx"] + 1, c["nely"] + 1, 3), np.uint8)
    m[:, 0] = 1
    return m.reshape(-1)


def _gradient_design(c, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.rand(c["nelz"], c["nelx"], c["nely"], dtype=torch.float64, device="cuda", generator=g)
    return (0.05 + 0.95 * x).permute(2, 1, 0)


def _density_inputs(c, seed):
    solid, void = _masks({**c, "masks": True})
    x = (0.5 + 0.3 * _field(_shape(c), seed)).clamp(0.0, 1.0)
    g = -torch.exp(1.5 * _field(_shape(c), seed + 7919))
    return (_fortran(x), _fortran(g), _fortran(torch.as_tensor(solid, device="cuda")),
            _fortran(torch.as_tensor(void, device="cuda")))


def _oc_inputs(c, seed):
    solid, void = _masks({**c, "masks": True})
    x = _design(c, seed, solid, void)
    dc = _fortran(-torch.exp(2.0 * _field(_shape(c), seed + 7919)))
    dv = _fortran(1.0 + 0.25 * torch.tanh(_field(_shape(c), seed + 15485863)))
    solid, void = (_fortran(torch.as_tensor(m, device="cuda")) for m in (solid, void))
    free = ~(solid | void)
    return x, dc, dv, solid, void, free, float(c["volfrac"] * int(free.sum()))


def prepare(case, seed):
    c = case
    from pytopo3d_b200.stiffness import lk_H8

    if c["kind"] == "top3d":
        from pytopo3d_b200.optimizer import top3d

        # a seeded obstacle (a void box away from the supports and the load) makes the run's own problem
        rng = np.random.default_rng(seed)
        ob = np.zeros(_shape(c), bool)
        x0 = int(rng.integers(c["nelx"] // 4, c["nelx"] // 2))
        y0, z0 = int(rng.integers(0, c["nely"] // 2)), int(rng.integers(c["nelz"] // 3, c["nelz"] // 2))
        ob[y0:y0 + c["nely"] // 3, x0:x0 + c["nelx"] // 5, z0:z0 + c["nelz"] // 4] = True
        return {"case": c, "top3d": top3d, "obstacle": ob}
    if c["kind"] == "loop":
        from pytopo3d_b200.optimizer import SimpLoop

        solid, void = _masks(c)
        x0 = _design(c, seed, solid, void)
        loop = SimpLoop(c["nelx"], c["nely"], c["nelz"], c["volfrac"], PENAL, c["rmin"], lk_H8(elem_size=1.0),
                        _edge_load(c), _fixed(c), solid, void, projection_eta=ETA, move=MOVE,
                        precision=c["precision"], x0=x0)
        return {"case": c, "loop": loop, "x0": loop.x.clone()}
    if c["kind"] == "gradient":
        from pytopo3d_b200.autograd import ComplianceProblem, compliance

        problem = ComplianceProblem(c["nelx"], c["nely"], c["nelz"], _load_cases(c), c["rmin"], c["beta"], eta=ETA,
                                    penal=PENAL, recompute=c["recompute"])
        return {"case": c, "compliance": compliance, "problem": problem, "x": _gradient_design(c, seed)}
    if c["kind"] == "batch":
        from pytopo3d_b200.batch import BatchRunner, batched_cantilevers

        specs = batched_cantilevers(c["designs"], c["spec_seed"])
        runner = BatchRunner(specs, precision="mixed", tune=None)
        runner.run(1)  # the graph is captured for designs whose solvers have run once
        x0 = []
        for k, (s, loop) in enumerate(zip(specs, runner.loops)):
            x = (s.volfrac * (1.0 + 0.7 * _field((s.nely, s.nelx, s.nelz), seed + 1000 * k))).clamp(0.02, 1.0)
            x = x.permute(2, 1, 0).contiguous().reshape(-1)
            x[loop.S.solid.bool()] = 1.0
            x[loop.S.void.bool()] = 0.0
            x0.append(x)
        return {"case": c, "runner": runner, "x0": x0}
    if c["kind"] == "density":
        from pytopo3d_b200 import apply_density_filter_chain_rule, build_filter, build_physical_density

        H, Hs = build_filter(c["nelx"], c["nely"], c["nelz"], c["rmin"])
        return {"case": c, "H": H, "Hs": Hs, "fwd": build_physical_density, "bwd": apply_density_filter_chain_rule,
                "in": _density_inputs(c, seed)}
    if c["kind"] == "oc":
        from pytopo3d_b200 import build_filter, optimality_criteria_update_projected

        H, Hs = build_filter(c["nelx"], c["nely"], c["nelz"], c["rmin"])
        return {"case": c, "H": H, "Hs": Hs, "oc": optimality_criteria_update_projected, "in": _oc_inputs(c, seed)}
    if c["kind"] == "solve":
        from pytopo3d_b200 import HexSolver

        solver = HexSolver(c["nelx"], c["nely"], c["nelz"], lk_H8(elem_size=1.0), _fixed(c),
                           precision=c["precision"])
        rho = _design(c, seed).permute(2, 1, 0).reshape(-1)
        return {"case": c, "solver": solver, "rho": rho, "F": torch.as_tensor(_edge_load(c)).cuda()}
    raise ValueError(c["kind"])


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _restart(loop, x0, beta):
    """The loop at the design x0 with no earlier solutions, as a continued run starts."""
    loop.x.copy_(x0)
    loop.S.U.zero_()
    loop.S.U_prev.zero_()
    loop.S.n_solved = 0
    loop.set_beta(beta)


def run(state):
    c = state["case"]
    if c["kind"] == "top3d":
        xphys, _, compliance, _ = state["top3d"](c["nelx"], c["nely"], c["nelz"], c["volfrac"], PENAL, c["rmin"], 0.5,
                                                 elem_size=1.0, obstacle_mask=state["obstacle"],
                                                 maxloop=c["maxloop"], beta_schedule=(1.0, 4.0))
        return {"physical": xphys, "compliance": compliance}
    if c["kind"] == "loop":
        loop = state["loop"]
        _restart(loop, state["x0"], c["beta"])
        cs = []
        for _ in range(c["steps"]):
            cs.append(loop.step()[:1])
        # displacements inside the 1e-9 voids are left out: the load does not determine them
        return {"design": loop.design(), "physical": loop.physical(), "gradient": loop.S.dc_dx,
                "compliance": torch.cat(cs)}
    if c["kind"] == "gradient":
        x = state["x"].detach().requires_grad_(True)
        value = state["compliance"](x, state["problem"])
        value.backward()
        return {"compliance": value.detach(), "gradient": x.grad}
    if c["kind"] == "batch":
        runner = state["runner"]
        for loop, x0 in zip(runner.loops, state["x0"]):
            _restart(loop, x0, 1.0)
        runner.run_graph(c["steps"])
        return {"design": [loop.x for loop in runner.loops], "compliance": np.asarray(runner.compliance)}
    if c["kind"] == "density":
        x, g, solid, void = state["in"]
        rf, rp, dp = state["fwd"](x, state["H"], state["Hs"], c["beta"], ETA, solid, void)
        return {"filtered": rf, "physical": rp, "dproj": dp, "dx": state["bwd"](g, dp, state["H"], state["Hs"])}
    if c["kind"] == "oc":
        x, dc, dv, solid, void, free, target = state["in"]
        x_new, rho = state["oc"](x, dc, dv, MOVE, target, state["H"], state["Hs"], c["beta"], ETA, free, solid, void)
        return {"design": x_new, "physical": rho}
    state["solver"].set_density(state["rho"], PENAL)
    return {"U": state["solver"].solve(state["F"])}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _taps(rmin):
    r = int(math.ceil(rmin))
    return [(dx, dy, dz, rmin - math.sqrt(dx * dx + dy * dy + dz * dz))
            for dx, dy, dz in itertools.product(range(-r, r + 1), repeat=3)
            if rmin - math.sqrt(dx * dx + dy * dy + dz * dz) > 1e-9]


def _size(c):
    nele = c["nelx"] * c["nely"] * c["nelz"]
    return nele, 3 * (c["nelx"] + 1) * (c["nely"] + 1) * (c["nelz"] + 1)


# one application of the operator: 8 corners of 24 multiply-adds of a 3-vector, with the
# symmetry of the element matrix used (279 operations a node)
_OP_FLOPS = 279.0


def work(case):
    """Each input read and each output written once; operations: an operator application
    for each solve and its residual, and the filter's taps for each filtering of the pass."""
    c = case
    if c["kind"] == "batch":
        from pytopo3d_b200.batch import batched_cantilevers

        out = {"bytes": 0.0, "flops": 0.0}
        for s in batched_cantilevers(c["designs"], c["spec_seed"]):
            w = work(_loop("", s.nelx, s.nely, s.nelz, "mixed", s.volfrac, s.rmin, 1.0, True, c["steps"]))
            out = {k: out[k] + w[k] for k in out}
        return out
    nele, ndof = _size(c)
    if c["kind"] == "solve":
        return {"bytes": 8.0 * (nele + 2 * ndof), "flops": 2 * _OP_FLOPS * ndof / 3}
    taps = 2.0 * len(_taps(c["rmin"])) * nele
    if c["kind"] == "density":
        return {"bytes": nele * (8.0 * 7 + 2), "flops": 2 * taps}  # x, g, Hs; rf, rp, dp, dx; masks
    if c["kind"] == "oc":
        return {"bytes": nele * (8.0 * 6 + 3), "flops": 2 * taps}  # x, dc, dv, Hs; x_new, rho; masks
    if c["kind"] == "gradient":
        return {"bytes": 8.0 * (3 * nele + 3 * ndof), "flops": 2 * taps + 6 * _OP_FLOPS * ndof / 3}
    steps = c["steps"] if c["kind"] == "loop" else 2 * c["maxloop"] + 2
    # design, Hs, masks in; design, density out; load in, displacements in and out
    return {"bytes": steps * (nele * (8.0 * 4 + 3) + 8.0 * 3 * ndof),
            "flops": steps * (5 * taps + 2 * _OP_FLOPS * ndof / 3)}


def tolerance(case):
    """About four times what other smoothing degrees and other summation orders show."""
    c = case
    if c["kind"] == "density":
        return {"rel": 1e-12, "max": 1e-10}  # 64-bit sums of up to a thousand taps
    if c["kind"] == "oc":
        return {"rel": 2e-8, "max": 1e-6}  # the bisection ends at a relative bracket of 1e-8
    mixed = c["kind"] == "batch" or c.get("precision") == "mixed"
    if mixed:
        return {"rel": 1.5e-5, "max": 2e-4}  # solves stop at a residual of 1e-6
    return {"rel": 2e-9, "max": 5e-7}  # solves stop at a residual of 1e-10


# ---------------------------------------------------------------------------
# a pass in plain 64-bit torch
# ---------------------------------------------------------------------------
def _element_stiffness():
    """Unit cube, E = 1, nu = 0.3, shear modulus 0.4, 2x2x2 Gauss points."""
    S = np.zeros((6, 6))
    S[:3, :3] = -0.3
    S[[0, 1, 2], [0, 1, 2]] = 1.0
    S[[3, 4, 5], [3, 4, 5]] = 1.0 / 0.4
    C = np.linalg.inv(S)
    sg = 2.0 * np.asarray(CORNERS, float) - 1.0
    KE = np.zeros((24, 24))
    for p in itertools.product((-1.0, 1.0), repeat=3):
        lin = 1.0 + sg * np.asarray(p) / math.sqrt(3.0)
        G = 0.25 * sg * np.stack([lin[:, 1] * lin[:, 2], lin[:, 0] * lin[:, 2], lin[:, 0] * lin[:, 1]], 1)
        B = np.zeros((6, 24))
        for k in range(3):
            B[k, k::3] = G[:, k]
        for row, (i, j) in zip((3, 4, 5), ((0, 1), (1, 2), (2, 0))):
            B[row, i::3], B[row, j::3] = G[:, j], G[:, i]
        KE += B.T @ C @ B / 8.0
    return torch.as_tensor(KE).cuda()


class _Plain:
    """Filter, elasticity and OC update on (nelz, nelx, nely) tensors."""

    def __init__(self, c, solid, void, rmin):
        self.c = c
        flat = lambda m: torch.as_tensor(np.ascontiguousarray(np.transpose(m, (2, 1, 0)))).cuda()
        self.solid, self.void = flat(solid), flat(void)
        self.free = ~(self.solid | self.void)
        self.taps = _taps(rmin)
        self.dims = (c["nelz"], c["nelx"], c["nely"])
        self.Hs = self.H(torch.ones(self.dims, dtype=torch.float64, device="cuda"))
        self.KE = _element_stiffness()
        e = torch.arange(c["nelx"] * c["nely"] * c["nelz"], device="cuda")
        y, x, z = e % c["nely"], (e // c["nely"]) % c["nelx"], e // (c["nely"] * c["nelx"])
        nodes = torch.stack([_node(c, x + ox, y + oy, z + oz) for ox, oy, oz in CORNERS], 1)
        self.edof = (3 * nodes[:, :, None] + torch.arange(3, device="cuda")).reshape(-1, 24)
        self.live = torch.as_tensor(_fixed(c)).cuda() == 0

    def H(self, v):
        r = int(max(abs(t[0]) for t in self.taps))
        p = torch.nn.functional.pad(v, (r,) * 6)
        nz, nx, ny = self.dims
        out = torch.zeros_like(v)
        for dx, dy, dz, w in self.taps:
            out += w * p[r + dz:r + dz + nz, r + dx:r + dx + nx, r + dy:r + dy + ny]
        return out

    def project(self, x, beta):
        rf = self.H(x) / self.Hs
        t = torch.tanh(beta * (rf - ETA))
        den = math.tanh(beta * ETA) + math.tanh(beta * (1.0 - ETA))
        rp = ((math.tanh(beta * ETA) + t) / den).clamp(0.0, 1.0)
        rp = torch.where(self.solid, 1.0, rp)
        rp = torch.where(self.void, 0.0, rp)
        return rf, rp, torch.where(self.free, beta * (1.0 - t * t) / den, 0.0)

    def chain(self, g, dproj):
        return self.H(g * dproj / self.Hs)

    def solve(self, rho, F, U0=None, rtol=1e-12):
        """Conjugate gradients with the diagonal as preconditioner, from U0."""
        E = (EMIN + (1.0 - EMIN) * rho.reshape(-1) ** PENAL)[:, None]

        def K(u):
            out = torch.zeros_like(u)
            return out.index_add_(0, self.edof.reshape(-1), ((u[self.edof] @ self.KE) * E).reshape(-1)) * self.live

        d = torch.zeros_like(F).index_add_(0, self.edof.reshape(-1), (E * self.KE.diagonal()).reshape(-1))
        u = torch.zeros_like(F) if U0 is None else U0.clone()
        for _ in range(4):  # the true residual again after each run
            r = (F - K(u)) * self.live
            z = r / d
            p, rz = z.clone(), torch.dot(r, z)
            for it in range(20000):
                q = K(p)
                alpha = rz / torch.dot(p, q)
                u += alpha * p
                r -= alpha * q
                z = r / d
                rz, old = torch.dot(r, z), rz
                p = z + (rz / old) * p
                if it % 50 == 49 and float(r.norm()) <= rtol * float(F.norm()):
                    break
        return u

    def energy(self, U):
        ue = U[self.edof]
        return ((ue @ self.KE) * ue).sum(1).reshape(self.dims)

    def sensitivities(self, rho, dproj, U):
        ce = self.energy(U)
        c = float(((EMIN + (1.0 - EMIN) * rho ** PENAL) * ce).sum())
        dc = -PENAL * (1.0 - EMIN) * rho ** (PENAL - 1.0) * ce
        return c, self.chain(dc, dproj), self.chain(self.free.double(), dproj)

    def oc(self, x, dc, dv, target, beta):
        ratio = torch.where(self.free, (-dc / dv.clamp(min=1e-20)).clamp(min=0.0), 0.0)
        ratio = ratio / ratio.max()
        lo, hi, best = 0.0, 1.0e12, (math.inf, None)
        for _ in range(80):
            lam = 0.5 * (lo + hi)
            xn = x * torch.sqrt((ratio / (lam + 1e-30)).clamp(min=1e-30))
            xn = torch.minimum(torch.maximum(xn, x - MOVE), x + MOVE).clamp(0.0, 1.0)
            xn = torch.where(self.solid, 1.0, torch.where(self.void, 0.0, xn))
            vol = float(self.project(xn, beta)[1][self.free].sum())
            if abs(vol - target) < best[0]:
                best = (abs(vol - target), xn)
            lo, hi = (lam, hi) if vol > target else (lo, lam)
            if (hi - lo) / (hi + lo) < 1e-8:
                break
        return best[1]

    def loop(self, x, beta, volfrac, steps, F):
        target, cs, U, dc = volfrac * int(self.free.sum()), [], None, None
        for _ in range(steps):
            _, rho, dproj = self.project(x, beta)
            U = self.solve(rho, F, U)
            c, dc, dv = self.sensitivities(rho, dproj, U)
            x = self.oc(x, dc, dv, target, beta)
            cs.append(c)
        return x, self.project(x, beta)[1], dc, cs


def _out(v):
    return v.permute(2, 1, 0)


def exact(case, seed):
    """What ``run`` returns, from the formulas; None where the plain solve takes too long."""
    c = case
    if c["kind"] in ("top3d", "batch"):
        return None
    nele = c["nelx"] * c["nely"] * c["nelz"]
    if c["kind"] in ("loop", "solve", "gradient") and nele > 80000:
        return None
    flat = lambda t: t.permute(2, 1, 0).contiguous()
    if c["kind"] == "loop":
        solid, void = _masks(c)
        P = _Plain(c, solid, void, c["rmin"])
        x, rho, dc, cs = P.loop(flat(_design(c, seed, solid, void)), c["beta"], c["volfrac"], c["steps"],
                               torch.as_tensor(_edge_load(c)).cuda())
        return {"design": _out(x), "physical": _out(rho), "gradient": dc.reshape(-1),
                "compliance": torch.tensor(cs, dtype=torch.float64)}
    none = np.zeros(_shape(c), bool)
    if c["kind"] == "gradient":
        P = _Plain(c, none, none, c["rmin"])
        _, rho, dproj = P.project(flat(_gradient_design(c, seed)), c["beta"])
        value, grad = 0.0, 0.0
        for F in torch.as_tensor(_load_cases(c)).cuda():
            U = P.solve(rho, F)
            value += float(torch.dot(F, U))
            grad = grad + P.sensitivities(rho, dproj, U)[1]
        return {"compliance": torch.tensor(value, dtype=torch.float64), "gradient": _out(grad)}
    if c["kind"] == "solve":
        P = _Plain(c, none, none, 1.0)
        return {"U": P.solve(flat(_design(c, seed)), torch.as_tensor(_edge_load(c)).cuda())}
    solid, void = _masks({**c, "masks": True})
    P = _Plain(c, solid, void, c["rmin"])
    if c["kind"] == "density":
        x, g, _, _ = _density_inputs(c, seed)
        rf, rp, dp = P.project(flat(x), c["beta"])
        return {"filtered": _out(rf), "physical": _out(rp), "dproj": _out(dp), "dx": _out(P.chain(flat(g), dp))}
    x, dc, dv, _, _, _, target = _oc_inputs(c, seed)
    xn = P.oc(flat(x), flat(dc), flat(dv), target, c["beta"])
    return {"design": _out(xn), "physical": _out(P.project(xn, c["beta"])[1])}
