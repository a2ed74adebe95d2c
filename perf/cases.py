"""What the framework is timed on.

Every case is a call that a program of this framework makes, through the C ABI
or its Python binding, over the range of sizes that the scenes, tests and the
benchmark of this repository use: from a 1,000-particle scene that is stepped
once per call up to the million-particle double dam break.

Kinds:
  frame     host state in (sph_set_state, sph_set_time), `steps` steps of one
            scene, host state out (sph_get_state) into pinned buffers: a
            program that edits or rewinds the fluid and advances it to the
            next picture
  batch     the same for many independent scenes in one context
  gradient  one iteration of an optimisation through the WCSPH step: state in,
            forward with checkpoints, backward, gradients out
  density   sph_density_noalloc on device buffers: densities for a caller that
            holds its particles on the GPU and may not allocate
"""
import ctypes as C
import math

import numpy as np
import torch

from sph2o_b200 import api, scenes

WCSPH, PCISPH, DFSPH = scenes.WCSPH, scenes.PCISPH, scenes.DFSPH


def listed():
    return [
        # the smallest scene of the tests, stepped once per call: an interactive
        # program that shows every step; all force models
        frame("step_wcsph_1k", WCSPH, (10, 10, 10), 0.025, 1, dt=1e-4, visc="xsph", st=0.05, adh=0.5),
        # the small dam break of the benchmark, 20 steps between pictures
        frame("frame_wcsph_8k", WCSPH, (20, 20, 20), 0.025, 20, dt=1e-4),
        # boundary particles with normals and collision (boundary method 1)
        frame("frame_dfsph_pcib_26k", DFSPH, (31, 29, 29), 0.0125, 4, dt=5e-4, boundary=1),
        # the water column with surface tension of the benchmark
        frame("frame_dfsph_st_125k", DFSPH, (50, 50, 50), 0.01, 4, dt=5e-4, st=0.05),
        # a viscous liquid that wets its tank: boundary viscosity, adhesion, an
        # odd particle count above the size where the kernels change their mapping
        frame("frame_wcsph_wet_306k", WCSPH, (71, 59, 73), 0.01, 5, dt=1e-4, visc="standard", bvisc=0.01, st=0.05,
              adh=0.5),
        # the headline scene of the benchmark, both solvers
        frame("frame_dfsph_1m", DFSPH, (100, 100, 50), 0.005, 4, dt=5e-4, double=True),
        frame("frame_pcisph_1m", PCISPH, (100, 100, 50), 0.005, 3, dt=2e-4, double=True),
        # many scenes at once: parameter studies, data sets of simulations
        {"name": "batch_wcsph_64", "kind": "batch", "method": WCSPH, "count": 64, "low": 2000, "high": 40000, "steps": 8},
        {"name": "batch_dfsph_24", "kind": "batch", "method": DFSPH, "count": 24, "low": 2000, "high": 40000, "steps": 3},
        # the differentiable workload: below and above the size where the adjoint changes its mapping
        {"name": "gradient_wcsph_33k", "kind": "gradient", "nx": 32, "ny": 32, "nz": 32, "radius": 0.02, "steps": 20,
         "every": 10, "bvisc": 0.0},
        {"name": "gradient_wcsph_91k", "kind": "gradient", "nx": 45, "ny": 47, "nz": 43, "radius": 0.02, "steps": 6,
         "every": 3, "bvisc": 0.01},
        # densities of particles that are on the GPU already
        {"name": "density_30k", "kind": "density", "nx": 31, "ny": 33, "nz": 29, "radius": 0.02},
    ]


def frame(name, method, dims, radius, steps, dt, visc="artificial", bvisc=0.0, st=0.0, adh=0.0, boundary=2,
          double=False):
    c = {"kind": "frame", "method": method, "nx": dims[0], "ny": dims[1], "nz": dims[2], "radius": radius,
         "steps": steps, "dt": dt, "viscosity_method": visc, "boundary_viscosity": bvisc, "surface_tension": st,
         "adhesion": adh, "boundary": boundary, "double": double}
    if name:
        c["name"] = name
    return c


def _dims(rng, low, high):
    """Lattice counts of a block of about exp(uniform) particles, sides within a factor of two."""
    n = math.exp(rng.uniform(math.log(low), math.log(high)))
    ax, ay = rng.uniform(0.6, 1.5), rng.uniform(0.6, 1.5)
    nz = (n / (ax * ay)) ** (1.0 / 3.0)
    return max(3, round(ax * nz)), max(3, round(ay * nz)), max(3, round(nz))


def _radius(n):
    """The particle radius that the repository's scenes use around n particles."""
    return 0.025 if n < 15000 else 0.02 if n < 60000 else 0.01 if n < 400000 else 0.005


def draw(rng):
    kind = rng.choice(["frame"] * 6 + ["batch", "gradient", "gradient", "density"])
    if kind == "frame":
        method = rng.choice([WCSPH, PCISPH, DFSPH])
        dims = _dims(rng, 700, 700000)
        n = dims[0] * dims[1] * dims[2]
        r = _radius(n)
        steps = max(1, min(20, int(rng.uniform(0.5, 1.0) * 4.0e6 / (n + 40000))))
        if method != WCSPH:
            steps = min(steps, 4)
        dt = {WCSPH: min(1e-4, 0.01 * r), PCISPH: min(2e-4, 0.04 * r), DFSPH: 5e-4}[method]
        visc = rng.choice(["artificial", "artificial", "xsph"] if method == DFSPH else ["artificial", "xsph", "standard"])
        boundary = rng.choice([2, 2, 2, 1]) if n < 60000 else 2
        return frame(None, method, dims, r, steps, dt, visc=visc, bvisc=rng.choice([0.0, 0.0, 0.01]),
                     st=rng.choice([0.0, 0.05]), adh=0.0 if boundary == 1 else rng.choice([0.0, 0.0, 0.5]),
                     boundary=boundary)
    if kind == "batch":
        method = rng.choice([WCSPH, DFSPH])
        low = int(math.exp(rng.uniform(math.log(1000), math.log(5000))))
        return {"kind": "batch", "method": method, "count": rng.randint(3, 48), "low": low,
                "high": int(low * rng.uniform(2.0, 8.0)), "steps": rng.randint(2, 8 if method == WCSPH else 3)}
    dims = _dims(rng, 1500, 100000 if kind == "gradient" else 60000)
    n = dims[0] * dims[1] * dims[2]
    c = {"kind": kind, "nx": dims[0], "ny": dims[1], "nz": dims[2], "radius": _radius(min(n, 50000))}
    if kind == "gradient":
        steps = rng.randint(4, 20 if n < 50000 else 6)
        c |= {"steps": steps, "every": rng.randint(2, steps), "bvisc": rng.choice([0.0, 0.01])}
    return c


# ---- inputs ---------------------------------------------------------------

VISC = {"standard": scenes.VISC_STANDARD, "artificial": scenes.VISC_ARTIFICIAL, "xsph": scenes.VISC_XSPH}


def scene_of(case, seed):
    """The scene of a single-scene case: a block (or the two of the double dam
    break) standing one particle spacing from the walls of its corner."""
    r = case["radius"]
    n = (case["nx"], case["ny"], case["nz"])
    if case["kind"] != "frame":
        ext = [2 * r * k for k in n]
        return scenes.scene(method=WCSPH, radius=r, blocks=[scenes.block(n, r, (2 * r,) * 3)],
                            tank=((0, 0, 0), (2 * ext[0] + 8 * r, ext[1] + 8 * r, ext[2] + 8 * r)), time_step=2e-4,
                            viscosity=0.01, boundary_viscosity=case.get("bvisc", 0.0), jitter=0.02, seed=seed)
    spheres, lo = [], (2 * r,) * 3
    if case["double"]:
        ext = [2 * r * k for k in n]
        tank = ((0, 0, 0), (4 * ext[0], 2 * ext[1], 4 * ext[2]))
        blocks = [scenes.block(n, r, lo), scenes.block(n, r, (tank[1][0] - 2 * r - ext[0], tank[1][1] - 2 * r - ext[1],
                                                              2 * r))]
        spheres = [((0.5 * tank[1][0], 0.5 * tank[1][1], 0.3), 0.2)]
    else:
        ext = [2 * r * k for k in n]
        tank = ((0, 0, 0), (2 * ext[0] + 8 * r, ext[1] + 8 * r, ext[2] + 8 * r))
        blocks = [scenes.block(n, r, lo)]
    if case["boundary"] == 1:
        tank = ((0, 0, 0), tuple(float(math.ceil(t)) for t in tank[1]))
    st, adh = case["surface_tension"], case["adhesion"]
    d = scenes.scene(method=case["method"], radius=r, blocks=blocks, tank=tank, spheres=spheres, time_step=case["dt"],
                     max_time_step=1e-3, eta=0.01 if case["method"] == PCISPH else 1e-4,
                     viscosity_method=VISC[case["viscosity_method"]],
                     viscosity=0.001 if case["viscosity_method"] == "standard" else 0.01,
                     boundary_viscosity=0.1 * case["boundary_viscosity"] if case["viscosity_method"] == "standard"
                     else case["boundary_viscosity"],
                     surface_tension_method=scenes.SURFACE_TENSION_AKINCI if st else -1, surface_tension=st,
                     adhesion_method=scenes.ADHESION_AKINCI if adh else -1, adhesion=adh, jitter=0.02, seed=seed)
    return scenes.with_pcisph_boundary(d) if case["boundary"] == 1 else d


def stirred(x, seed, speed):
    """A flow in motion: a horizontal eddy over the fluid (divergence free), a
    fall, and a little noise."""
    lo, hi = x.min(0), x.max(0)
    ext = np.maximum(hi - lo, 1e-6)
    q = (x - lo) / ext * np.float32(math.pi)
    rng = np.random.default_rng(seed)
    v = rng.normal(0.0, 0.002 * speed, x.shape).astype(np.float32)
    v[:, 0] += speed * np.sin(q[:, 0]) * np.cos(q[:, 1])
    v[:, 1] -= speed * (ext[1] / ext[0]) * np.cos(q[:, 0]) * np.sin(q[:, 1])
    return np.ascontiguousarray(v, np.float32)


def batch_scenes_of(case, seed):
    rng = np.random.default_rng(seed)
    size = np.random.default_rng(11)  # the sizes belong to the case, the particles to the seed
    r, out = 0.01, []
    for i in range(case["count"]):
        nf = math.exp(size.uniform(math.log(case["low"]), math.log(case["high"])))
        ax, ay = size.uniform(0.5, 2.0, 2)
        nz = (nf / (ax * ay)) ** (1.0 / 3.0)
        n = (max(2, round(ax * nz)), max(2, round(ay * nz)), max(2, round(nz)))
        ext = [2 * r * k for k in n]
        out.append(scenes.scene(method=case["method"], radius=r, blocks=[scenes.block(n, r, (2 * r,) * 3)],
                                tank=((0, 0, 0), (max(1.0, 2 * ext[0] + 8 * r), max(1.0, ext[1] + 8 * r),
                                                  max(1.0, ext[2] + 8 * r))),
                                time_step=1e-4, viscosity=float(rng.uniform(0.005, 0.05)), eta=1e-3, eta_v=1e-3,
                                jitter=0.02, seed=int(rng.integers(1 << 30))))
    return out


def pinned(n, cols):
    return torch.empty((n, cols) if cols > 1 else (n,), dtype=torch.float32, pin_memory=True).numpy()


def to_pinned(a):
    out = pinned(a.shape[0], a.shape[1])
    out[...] = a
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        sc = [api.Scene.from_dict(d) for d in batch_scenes_of(case, seed)]
        vels = [stirred(s.fluid()[0], seed + i, 0.5) for i, s in enumerate(sc)]
        sim = api.Batch(sc, vels=vels)
        x = np.concatenate([s.fluid()[0] for s in sc])
        return {"kind": kind, "sim": sim, "steps": case["steps"], "x": to_pinned(x), "v": to_pinned(np.concatenate(vels)),
                "out": (pinned(sim.nf, 3), pinned(sim.nf, 3), pinned(sim.nf, 1))}
    sc = api.Scene.from_dict(scene_of(case, seed))
    x = sc.fluid()[0]
    if kind == "density":
        d, b = sc.desc(), sc.boundary()
        lo = np.minimum(b.min(0), x.min(0)).astype(np.float32)
        hi = np.maximum(b.max(0), x.max(0)).astype(np.float32)
        psi = np.full((b.shape[0], 1), d.density0 * 0.75 * (2 * d.particle_radius) ** 3, np.float32)
        fn = api.lib().sph_density_noalloc
        fn.restype = C.c_int
        fn.argtypes = [C.c_float, C.c_float, C.c_void_p, C.c_uint, C.c_void_p, C.c_uint, C.POINTER(C.c_float),
                       C.POINTER(C.c_float), C.c_void_p, C.c_void_p]
        rho = torch.empty(x.shape[0], dtype=torch.float32, device="cuda")
        return {"kind": kind, "fn": fn, "r": d.particle_radius, "rho0": d.density0, "x": torch.from_numpy(x).cuda(),
                "b": torch.from_numpy(np.concatenate([b, psi], 1)).cuda(), "lo": (C.c_float * 3)(*lo),
                "hi": (C.c_float * 3)(*hi), "rho": rho}
    if kind == "gradient":
        v, target = scenes.adjoint_problem(x, seed_v=seed, seed_t=seed + 1)
        return {"kind": kind, "sim": api.Simulation.from_scene(sc, vel=v), "x": x, "v": v, "target": target,
                "steps": case["steps"], "every": case["every"]}
    v = stirred(x, seed, speed_of(case))
    sim = api.Simulation.from_scene(sc, vel=v)
    return {"kind": kind, "sim": sim, "steps": case["steps"], "dt": case["dt"], "x": to_pinned(x), "v": to_pinned(v),
            "out": (pinned(sim.nf, 3), pinned(sim.nf, 3), pinned(sim.nf, 1))}


def speed_of(case):
    return 1.0 if case["method"] != WCSPH else 0.5


def _f(a):
    return a.ctypes.data_as(C.POINTER(C.c_float))


def run(state):
    kind = state["kind"]
    if kind == "density":
        rc = state["fn"](state["r"], state["rho0"], state["x"].data_ptr(), state["x"].shape[0], state["b"].data_ptr(),
                         state["b"].shape[0], state["lo"], state["hi"], state["rho"].data_ptr(),
                         torch.cuda.current_stream().cuda_stream)
        if rc != 0:
            raise RuntimeError("sph_density_noalloc: %d" % rc)
        return state["rho"]
    sim = state["sim"]
    sim.set_state(state["x"], state["v"])
    if kind == "gradient":
        loss = sim.wcsph_forward(state["steps"], state["target"], ckpt_every=state["every"])
        return {"loss": loss, **sim.wcsph_backward(want_x0=True)}
    if kind == "frame":
        sim.set_time(0.0, state["dt"])
    sim.step(state["steps"])
    x, v, rho = state["out"]
    sim._check(api.lib().sph_get_state(sim._h, _f(x), _f(v), _f(rho)))
    return {"x": x, "v": v, "rho": rho}


def work(case):
    """Bytes: the state that goes in and comes out, and for each step the state
    once through memory. Operations: about 30 neighbours a particle, about 20
    operations for each pair and pass over the neighbours."""
    if case["kind"] == "batch":
        size, n = np.random.default_rng(11), 0.0
        for _ in range(case["count"]):
            n += math.exp(size.uniform(math.log(case["low"]), math.log(case["high"])))
            size.uniform(0.5, 2.0, 2)
    else:
        n = case["nx"] * case["ny"] * case["nz"] * (2 if case.get("double") else 1)
    steps = case.get("steps", 1)
    passes = 1 if case["kind"] == "density" else 3 + 6 if case["kind"] == "gradient" else \
        {WCSPH: 2, PCISPH: 2 + 4, DFSPH: 2 + 6 + 3}[case["method"]]
    state = 16 if case["kind"] == "density" else 52
    return {"bytes": n * state * (1 + (steps if case["kind"] != "density" else 0)), "flops": n * 30 * 20 * passes * steps}


# ---- the same in 64 bits, in torch ----------------------------------------

def pairs(x, y, h, reach=None):
    """(i, j) with |x_i - y_j| <= reach (h if not given) among the 27 cells of edge h around x_i's."""
    reach = reach or h
    dev = x.device
    cx, cy = torch.floor(x / h).long(), torch.floor(y / h).long()
    lo = torch.minimum(cx.min(0).values, cy.min(0).values) - 1
    dim = torch.maximum(cx.max(0).values, cy.max(0).values) - lo + 2
    key = lambda c: ((c[:, 0] - lo[0]) * dim[1] + (c[:, 1] - lo[1])) * dim[2] + (c[:, 2] - lo[2])  # noqa: E731
    ky, order = torch.sort(key(cy))
    kx = key(cx)
    found = []
    step = 1 << 17
    for a in range(0, x.shape[0], step):
        k = kx[a:a + step]
        for dx in (-1, 0, 1):
            for dy in (-1, 0, 1):
                row = k + (dx * dim[1] + dy) * dim[2]
                s, e = torch.searchsorted(ky, row - 1), torch.searchsorted(ky, row + 1, right=True)
                cnt = e - s
                i = torch.repeat_interleave(torch.arange(k.shape[0], device=dev), cnt)
                off = torch.arange(i.shape[0], device=dev) - (torch.cumsum(cnt, 0) - cnt)[i]
                j = order[s[i] + off]
                i = i + a
                keep = (x[i] - y[j]).square().sum(1) <= reach * reach
                found.append(torch.stack([i[keep], j[keep]]))
    p = torch.cat(found, 1)
    return p[0], p[1]


class Fluid:
    """One scene in 64 bits: what SPH2O's solvers compute (SPHSolver.cpp, WCSPHSolver.cpp, PCISPHSolver.cpp,
    DFSPHSolver.cpp and the non-pressure forces), pair by pair. `visc`, `stiff` may carry gradients."""

    def __init__(self, desc, x, v, b, normals=None):
        d = self.d = desc
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev).double()  # noqa: E731
        self.x, self.v, self.b = t(x), t(v), t(b)
        r = float(d.particle_radius)
        self.h, self.m, self.rho0 = 4 * r, float(d.density0) * (2 * r) ** 3, float(d.density0)
        self.g = torch.tensor(list(d.gravity), dtype=torch.float64, device=dev)
        self.visc, self.stiff = float(d.viscosity), float(d.stiffness)
        self.pcib = d.boundary_method == 1
        self.dt, self.its, self.itsv = float(d.time_step), 0, 0
        self.n = self.x.shape[0]
        self.kws = self.kvws = torch.zeros(self.n, dtype=torch.float64, device=dev)
        self.normal = torch.zeros_like(self.x)
        if self.pcib:
            self.psi = torch.full((self.b.shape[0],), self.m, dtype=torch.float64, device=dev)
            self.bn, self.nf, self.tf = t(normals[0]), float(normals[1]), float(normals[2])
        elif self.b.shape[0]:
            i, j = pairs(self.b, self.b, self.h)
            self.psi = self.rho0 / self.add(self.b.shape[0], i, self.W((self.b[i] - self.b[j]).norm(dim=1)))
        else:
            self.psi = torch.zeros(0, dtype=torch.float64, device=dev)

    @staticmethod
    def add(n, i, w):
        return torch.zeros((n,) + w.shape[1:], dtype=w.dtype, device=w.device).index_add(0, i, w)

    def W(self, rl):
        q = rl / self.h
        w = torch.where(q <= 0.5, 6 * q ** 3 - 6 * q ** 2 + 1, 2 * (1 - q).clamp(min=0) ** 3)
        return 8 / (math.pi * self.h ** 3) * w

    def F(self, rl):
        """gradW(r) = F(|r|) r."""
        q, l = rl / self.h, 48 / (math.pi * self.h ** 3)
        f = torch.where(q <= 0.5, l / self.h ** 2 * (3 * q - 2), -l / self.h * (1 - q).clamp(min=0) ** 2 / rl)
        return torch.where(rl > 1e-9, f, torch.zeros_like(f))

    def search(self):
        with torch.no_grad():
            i, j = pairs(self.x, self.x, self.h)
            self.near = self.add(self.n, i, torch.ones_like(i, dtype=torch.float64))
            other = i != j  # a particle alone with itself: its own term is a constant
            self.i, self.j = i[other], j[other]
            self.ib, self.jb = pairs(self.x, self.b, self.h) if self.b.shape[0] else (self.i[:0], self.i[:0])
            self.near += self.add(self.n, self.ib, torch.ones_like(self.ib, dtype=torch.float64))
        self.geometry()

    def geometry(self):
        self.r = self.x[self.i] - self.x[self.j]
        self.rl = self.r.norm(dim=1)
        self.rb = self.x[self.ib] - self.b[self.jb]
        self.rbl = self.rb.norm(dim=1)
        self.G = self.F(self.rl)[:, None] * self.r
        self.Gb = self.F(self.rbl)[:, None] * self.rb

    def density(self):
        own = self.m * 8 / (math.pi * self.h ** 3)
        self.rho = own + self.add(self.n, self.i, self.m * self.W(self.rl)) + \
            self.add(self.n, self.ib, self.psi[self.jb] * self.W(self.rbl))

    def tait(self, rho):
        d = self.d
        return (self.stiff * self.rho0 / float(d.gamma) * ((rho / self.rho0) ** float(d.gamma) - 1)).clamp(min=0)

    def forces(self, pressure=False):
        d, m, i, j, ib, jb, rho = self.d, self.m, self.i, self.j, self.ib, self.jb, self.rho
        a = torch.zeros_like(self.x)
        if pressure:
            self.p = self.tait(rho)
            A, B = self.p / rho ** 2, self.p / self.rho0 ** 2
            a = a - self.add(self.n, i, (m * (A[i] + A[j]))[:, None] * self.G)
            if self.pcib:
                i2, j2 = pairs(self.b, self.x, self.h)
                i3, j3 = pairs(self.b, self.b, self.h)
                rb = self.add(self.b.shape[0], i2, self.m * self.W((self.b[i2] - self.x[j2]).norm(dim=1))) + \
                    self.add(self.b.shape[0], i3, self.m * self.W((self.b[i3] - self.b[j3]).norm(dim=1)))
                Bb = (self.tait(rb) / rb ** 2)[jb]
            else:
                Bb = B[ib]
            a = a - self.add(self.n, ib, (self.psi[jb] * (A[ib] + Bb))[:, None] * self.Gb)
        bv = 0.0 if self.pcib else float(d.boundary_viscosity)
        dv, vm = self.v[i] - self.v[j], d.viscosity_method
        if vm == 1:
            s = self.rl ** 2 + 0.01 * self.h ** 2
            a = a + self.add(self.n, i, (self.visc * m / rho[j] * (dv * self.r).sum(1) / s)[:, None] * self.G)
            if bv:
                s = self.rbl ** 2 + 0.01 * self.h ** 2
                a = a + self.add(self.n, ib, (bv * self.psi[jb] / rho[ib] * (self.v[ib] * self.rb).sum(1) / s)[:, None] *
                                 self.Gb)
        elif vm == 0:
            lap = lambda rl: 45 / (math.pi * self.h ** 6) * (self.h - rl).clamp(min=0)  # noqa: E731
            a = a - (self.visc / rho)[:, None] * self.add(self.n, i, (m / rho[j] * lap(self.rl))[:, None] * dv)
            if bv:
                a = a - (bv / rho)[:, None] * self.add(self.n, ib, (self.psi[jb] / rho[ib] * lap(self.rbl))[:, None] *
                                                       self.v[ib])
        elif vm == 2:
            a = a - self.add(self.n, i, (self.visc * m / rho[j] * self.W(self.rl) / self.dt)[:, None] * dv)
            if bv:
                a = a - self.add(self.n, ib, (bv * self.psi[jb] / rho[ib] * self.W(self.rbl) / self.dt)[:, None] *
                                 self.v[ib])
        if d.surface_tension_method == 3 and d.surface_tension:
            h, rl, st = self.h, self.rl, float(d.surface_tension)
            self.normal = nrm = h * self.add(self.n, i, (m / rho[j])[:, None] * self.G)
            c = 32 / math.pi / h ** 9
            w = (h - rl).clamp(min=0) ** 3 * rl ** 3
            coh = torch.where(2 * rl > h, c * w, 2 * c * w - h ** 6 / 64)
            kij = 2 * self.rho0 / (rho[i] + rho[j])
            a = a - self.add(self.n, i, kij[:, None] * (st * (m * coh / rl)[:, None] * self.r + st * (nrm[i] - nrm[j])))
        if d.adhesion_method == 4 and d.adhesion:
            h, rl = self.h, self.rbl
            w = (-4 * rl ** 2 / h + 6 * rl - 2 * h).clamp(min=0) ** 0.25
            w = torch.where(2 * rl > h, w, torch.zeros_like(w))
            a = a - self.add(self.n, ib, (float(d.adhesion) * self.psi[jb] * w / rl)[:, None] * self.rb)
        return a

    def collide(self, x, y):
        """PCISPH boundary particles: (x pushed out, normals) with the weights taken at y."""
        i, j = pairs(x, self.b, self.h, 0.5 * self.h)
        gap = 0.5 * self.h - (y[i] - self.b[j]).norm(dim=1)
        w = (gap / (0.5 * self.h)).clamp(min=0)
        ws, w2 = self.add(self.n, i, w), self.add(self.n, i, w * gap)
        avg = self.add(self.n, i, w[:, None] * self.bn[j])
        n = avg / avg.norm(dim=1, keepdim=True)
        return torch.where((ws > 0)[:, None], n, torch.zeros_like(n)), torch.where(ws > 0, w2 / ws, torch.zeros_like(ws))

    def bounce(self, n, u, v):
        d = (u * n).sum(1, keepdim=True) * n
        return torch.where((n.norm(dim=1) > 0)[:, None], self.tf * (u - d) - self.nf * d, v)

    def step_wcsph(self):
        self.search()
        self.density()
        a = self.forces(pressure=True) + self.g
        self.v = self.v + a * self.dt
        self.x = self.x + self.v * self.dt
        if self.pcib:
            n, s = self.collide(self.x, self.x)
            self.x = self.x + s[:, None] * n
            self.v = self.bounce(n, self.v, self.v)

    def step_pcisph(self, avg):
        d, dt = self.d, self.dt
        self.search()
        self.density()
        a = self.forces()
        ci, cj = pairs(self.x, self.x, self.h, 1.3 * self.h)
        bi, bj = pairs(self.x, self.b, self.h, 1.3 * self.h)
        ax = torch.arange(-1, 2, dtype=torch.float64, device=self.x.device) * (self.h / 2)
        lat = torch.cartesian_prod(ax, ax, ax)
        g = self.F(lat.norm(dim=1))[:, None] * lat
        beta = 2 * (self.m * float(d.time_step) / self.rho0) ** 2
        delta = 1 / (beta * float(g.sum(0).square().sum() + g.square().sum()))
        p, pa, it = torch.zeros_like(self.rho), torch.zeros_like(self.x), 0
        while (avg > float(d.eta) or it < d.min_iterations) and it < d.max_iterations:
            pv = self.v + (a + pa + self.g) * dt
            px = self.x + pv * dt
            if self.pcib:
                n, s = self.collide(self.x, px)
                px = px + s[:, None] * n
            self.rho = self.add(self.n, ci, self.m * self.W((px[ci] - px[cj]).norm(dim=1))) + \
                self.add(self.n, bi, self.psi[bj] * self.W((px[bi] - self.b[bj]).norm(dim=1)))
            err = (self.rho - self.rho0).clamp(min=0)
            p = p + delta * err
            avg = float((err / self.rho0).mean())
            A = p / self.rho ** 2
            pa = -self.add(self.n, self.i, (self.m * (A[self.i] + A[self.j]))[:, None] * self.G)
            if self.b.shape[0]:
                pa = pa - self.add(self.n, self.ib, (self.psi[self.jb] * A[self.ib])[:, None] * self.Gb)
            it += 1
        self.v = self.v + (a + self.g + pa) * dt
        self.x = self.x + self.v * dt
        return avg

    def change(self, v):
        return self.add(self.n, self.i, self.m * (self.G * (v[self.i] - v[self.j])).sum(1)) + \
            self.add(self.n, self.ib, self.psi[self.jb] * (self.Gb * v[self.ib]).sum(1))

    def corrected(self, v, k):
        ks = k[self.i] + k[self.j]
        ks = torch.where(ks.abs() > 1e-5, ks, torch.zeros_like(ks))
        kb = torch.where(k.abs() > 1e-5, k, torch.zeros_like(k))[self.ib]
        return v - self.dt * (self.add(self.n, self.i, (self.m * ks)[:, None] * self.G) +
                              self.add(self.n, self.ib, (self.psi[self.jb] * kb)[:, None] * self.Gb))

    def density_alpha(self):
        self.density()
        mg = self.m * self.G
        den = (self.add(self.n, self.i, mg) + self.add(self.n, self.ib, self.psi[self.jb, None] * self.Gb)).square().sum(1) + \
            self.add(self.n, self.i, mg.square().sum(1))
        self.alpha = torch.where(den > 1e-5, self.rho / den, torch.zeros_like(den))

    def step_dfsph(self):
        d = self.d
        a = self.forces()
        vmax = max(float((self.v + (a + self.g) * self.dt).norm(dim=1).max()), 1e-9)
        its = max(self.its, self.itsv)
        dt = self.dt * (0.9 if its > 6 else 1.05 if its < 4 else 1.0)
        dt = min(dt, float(d.cfl_factor) * 0.4 * 2 * float(d.particle_radius) / vmax)
        self.dt = dt = min(max(dt, min(1 / float(d.fps), float(d.min_time_step))), float(d.max_time_step))
        v = self.v + (a + self.g) * dt
        if self.pcib:
            v = self.bounce(self.normal, v, v)
        predicted = lambda v: (self.rho + dt * self.change(v)).clamp(min=self.rho0)  # noqa: E731
        v = self.corrected(v, torch.where(predicted(v) > self.rho0, self.kws / dt ** 2, 0.0))
        total, it, avg = torch.zeros_like(self.rho), 0, 0.0
        while (avg > float(d.eta) or it < d.min_iterations) and it < d.max_iterations:
            r = predicted(v) - self.rho0
            k = r * self.alpha / (dt ** 2 * self.rho)
            avg, total, it = float((r / self.rho0).mean()), total + k, it + 1
            v = self.corrected(v, k)
        self.kws, self.its = total * dt ** 2, it
        self.x = self.x + v * dt
        if self.pcib:
            self.normal, s = self.collide(self.x, self.x)
            self.x = self.x + s[:, None] * self.normal
        self.search()
        self.density_alpha()
        error = lambda v: torch.where(self.near < 20, 0.0, self.change(v).clamp(min=0))  # noqa: E731
        v = self.corrected(v, torch.where(error(v) > 0, self.kvws / dt, 0.0))
        total, it, avg = torch.zeros_like(self.rho), 0, 0.0
        while (avg > float(d.eta_v) / dt or it < d.min_iterations_v) and it < d.max_iterations:
            r = error(v)
            k = r * self.alpha / (dt * self.rho)
            avg, total, it = float((r / self.rho0).mean()), total + k, it + 1
            v = self.corrected(v, k)
        self.kvws, self.itsv, self.v = total * dt, it, v

    def run(self, steps):
        avg = 0.0
        if self.d.simulation_method == DFSPH:
            self.search()
            self.density_alpha()
        for _ in range(steps):
            if self.d.simulation_method == WCSPH:
                self.step_wcsph()
            elif self.d.simulation_method == PCISPH:
                avg = self.step_pcisph(avg)
            else:
                self.step_dfsph()
        return self.x, self.v, self.rho


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        got = []
        for i, d in enumerate(batch_scenes_of(case, seed)):
            sc = api.Scene.from_dict(d)
            x = sc.fluid()[0]
            got.append(Fluid(sc.desc(), x, stirred(x, seed + i, 0.5), sc.boundary()).run(case["steps"]))
        return {k: torch.cat([g[n] for g in got]) for n, k in enumerate(("x", "v", "rho"))}
    sc = api.Scene.from_dict(scene_of(case, seed))
    x, b, d = sc.fluid()[0], sc.boundary(), sc.desc()
    if kind == "density":
        f = Fluid(d, x, x, b[:0])
        f.b = torch.from_numpy(b).to(f.x.device).double()
        psi = np.float32(d.density0 * 0.75 * (2 * d.particle_radius) ** 3)
        f.psi = torch.full((b.shape[0],), float(psi), dtype=torch.float64, device=f.x.device)
        f.search()
        f.density()
        return f.rho
    if kind == "gradient":
        v, target = scenes.adjoint_problem(x, seed_v=seed, seed_t=seed + 1)
        f = Fluid(d, x, v, b)
        x0, v0 = f.x.requires_grad_(), f.v.requires_grad_()
        f.visc = torch.tensor(f.visc, dtype=torch.float64, device=x0.device, requires_grad=True)
        f.stiff = torch.tensor(f.stiff, dtype=torch.float64, device=x0.device, requires_grad=True)
        visc, stiff = f.visc, f.stiff
        xT, _, _ = f.run(case["steps"])
        loss = (xT - torch.from_numpy(target).to(xT.device).double()).square().sum() / f.n
        gx, gv, gn, gk = torch.autograd.grad(loss, (x0, v0, visc, stiff))
        return {"loss": float(loss.detach()), "v0": gv, "viscosity": float(gn), "stiffness": float(gk), "x0": gx}
    f = Fluid(d, x, stirred(x, seed, speed_of(case)), b, sc.boundary_normals())
    if f.pcib and case["method"] == PCISPH:
        return None  # its boundary particles have pressures of their own
    x, v, rho = f.run(case["steps"])
    return {"x": x, "v": v, "rho": rho}
