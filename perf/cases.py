"""Workloads of the explicit MPM step, each one pass through the public entry points.

A case names a scene (mesh, body, particles per cell, basis, transfer, material),
a precision form and the call a program makes on it:

  step      runtime.step: `steps` fused steps in one call
  loop      the hand-written loop body: update(partition), P2G, G2P
  adaptive  runtime.adaptive_steps: a time step from the particles' wave speed,
            read back on the host, before every step (the Taylor impact's loop)
  host      runtime.rollout_host: `steps` steps on host (pinned) buffers
  grad      runtime.rollout_grad: a taped rollout of `steps` steps and its
            gradients with respect to the initial velocities (and log E)

The precision forms are those of the library: "f64", "f32" (FP32 state, FP64 F)
and "f32x64" (FP32 state with FP64 positions). Particles start in a smoothly
deformed state with consistent stresses, so every term of the step is at work.
`exact` is the same step written in plain torch in FP64.
"""
import importlib.util
import math
import pathlib
import random
import sys

import torch
import torch.utils.checkpoint

ROOT = pathlib.Path(__file__).resolve().parent.parent
DEV = "cuda"
F64 = torch.float64


def package():
    """The package, whose folder name is no Python identifier."""
    if "tesserae_b200" in sys.modules:
        return sys.modules["tesserae_b200"]
    pkg = ROOT / "tesserae.jl_b200"
    spec = importlib.util.spec_from_file_location("tesserae_b200", pkg / "__init__.py",
                                                  submodule_search_locations=[str(pkg)])
    mod = importlib.util.module_from_spec(spec)
    sys.modules["tesserae_b200"] = mod
    spec.loader.exec_module(mod)
    return mod


# --------------------------------------------------------------------------
# cases
# --------------------------------------------------------------------------

def case(name, kind, cells, body, form, steps, ppc=2, basis="bspline", transfer="flip", material="neo", order="block",
         alpha=1.0, count=0):
    c = {"kind": kind, "nx": cells[0], "ny": cells[1], "nz": cells[2] if len(cells) == 3 else 0, "body": body,
         "form": form, "steps": steps, "ppc": ppc, "basis": basis, "transfer": transfer, "material": material,
         "order": order, "alpha": alpha, "count": count}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the README's two colliding disks, one step per call: a program that
        # looks at the state after every step; 10k particles, all latency
        case("disks2d_call", "step", (100, 100), "disks", "f64", 1, order="lattice"),
        # a 2D MLS-MPM (WLS + APIC) run between two outputs, on a ragged mesh
        case("mlsmpm2d_fused", "step", (257, 193), "block", "f32", 25, ppc=3, basis="wls_bspline", transfer="apic"),
        # the headline scene: 256^3 cells, 16.8 M particles in block order,
        # FP32 state with FP64 positions, several steps per call
        case("cube3d_fused", "step", (256, 256, 256), "block", "f32x64", 3),
        # the drop-in FP64 form on an odd mesh, particles as generated, a step per call
        case("block3d_f64_call", "step", (89, 103, 97), "block", "f64", 1, order="lattice"),
        # 64 particles per cell with per-particle Lame parameters (1.9 M particles)
        case("sphere3d_dense", "step", (64, 64, 64), "sphere", "f32x64", 8, ppc=4, order="lattice"),
        # Gaussian clusters with lognormal masses: blocks from empty to crowded
        case("clusters3d", "step", (256, 256, 256), "clusters", "f32x64", 2, count=4194304),
        # the Taylor impact: KernelCorrection weights, von Mises plasticity, a
        # slip floor, the time step from the particles at every step (1.48 M)
        case("taylor3d_adaptive", "adaptive", (72, 72, 134), "rod", "f32", 4, ppc=3, basis="kc_bspline",
             material="vonmises", order="lattice"),
        # the dam break (WLS(uGIMP), APIC, fluid, slip walls) at half resolution:
        # 18 M particles, the costliest step of the configurations
        case("dambreak3d", "step", (192, 192, 192), "column", "f32x64", 1, basis="wls_ugimp", transfer="apic",
             material="fluid"),
        # a loop written by hand with the verbs (custom work between them)
        case("verbs3d_loop", "loop", (75, 66, 81), "sphere", "f32", 1, ppc=3, basis="ugimp", order="lattice",
             alpha=0.98),
        # a host program without device arrays
        case("host3d_rollout", "host", (64, 64, 64), "block", "f32x64", 10),
        # inverse problems: gradients of a rollout loss with respect to v0 and
        # log E (the differentiable sphere), and through the dam break's step
        case("grad3d_sphere", "grad", (48, 48, 48), "sphere", "f32x64", 4, ppc=4, order="lattice"),
        case("grad3d_dambreak", "grad", (48, 48, 48), "column", "f32x64", 2, basis="wls_ugimp", transfer="apic",
             material="fluid"),
    ]


def draw(rng: random.Random):
    """One more case of the ranges above: meshes of 24 to about 200 cells per axis
    in 3D (40 to 400 in 2D), 1 to 25 steps per call, every basis, transfer and
    precision form in use."""
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def cells3(lo, hi):
        a = logint(lo, hi)
        return tuple(max(16, int(round(a * rng.uniform(0.8, 1.2)))) for _ in range(3))

    order = rng.choice(["block", "lattice"])
    form = rng.choice(["f64", "f32", "f32x64"])
    kind = rng.choice(["disks", "plane2d", "cube", "cube", "sphere", "clusters", "taylor", "dam", "loop", "host",
                       "grad", "gradgen"])
    if kind == "disks":
        a = logint(40, 400)
        return case(None, "step", (a, int(a * rng.uniform(0.9, 1.1))), "disks", rng.choice(["f64", "f32"]),
                    rng.choice([1, 1, 5]), ppc=rng.choice([2, 3]), basis=rng.choice(["bspline", "ugimp"]), order=order)
    if kind == "plane2d":
        a = logint(60, 400)
        return case(None, "step", (a, int(a * rng.uniform(0.7, 1.3))), "block", rng.choice(["f64", "f32"]),
                    logint(1, 25), ppc=rng.choice([2, 3]), basis="wls_bspline", transfer="apic", order=order)
    if kind == "cube":
        return case(None, "step", cells3(24, 180), "block", form, logint(1, 6),
                    basis=rng.choice(["bspline", "bspline", "ugimp"]), order=order, alpha=rng.choice([1.0, 0.98]))
    if kind == "sphere":
        return case(None, "step", cells3(24, 80), "sphere", form, logint(1, 8), ppc=rng.choice([3, 4]), order=order)
    if kind == "clusters":
        return case(None, "step", cells3(64, 200), "clusters", form, logint(1, 3), count=logint(100000, 4000000))
    if kind == "taylor":
        r = rng.choice([5, 6, 8, 9, 10, 12])
        return case(None, "adaptive", (6 * r, 6 * r, int(math.ceil(11.1375 * r))), "rod",
                    rng.choice(["f64", "f32"]), logint(1, 4), ppc=3, basis="kc_bspline", material="vonmises",
                    order="lattice")
    if kind == "dam":
        return case(None, "step", cells3(24, 130), "column", form, logint(1, 3),
                    basis=rng.choice(["wls_ugimp", "wls_bspline"]), transfer="apic",
                    material=rng.choice(["fluid", "neo"]), order=order)
    if kind == "loop":
        return case(None, "loop", cells3(24, 90), rng.choice(["sphere", "block"]), rng.choice(["f64", "f32"]), 1,
                    ppc=rng.choice([2, 3]), basis=rng.choice(["bspline", "ugimp"]), order=order,
                    alpha=rng.choice([1.0, 0.98]))
    if kind == "host":
        return case(None, "host", cells3(24, 70), "block", form, logint(1, 10), order=order)
    if kind == "grad":
        return case(None, "grad", cells3(20, 48), "sphere", form, logint(1, 5), ppc=rng.choice([3, 4]),
                    basis=rng.choice(["bspline", "ugimp"]), order=order)
    return case(None, "grad", cells3(20, 48), "column", form, logint(1, 2),
                basis=rng.choice(["wls_ugimp", "wls_bspline"]), transfer="apic", material="fluid", order=order)


# --------------------------------------------------------------------------
# scenes
# --------------------------------------------------------------------------

class Scene:
    """Mesh, step parameters and the host-side description of one case."""

    def __init__(self, c):
        self.c = c
        self.dim = 3 if c["nz"] else 2
        self.cells = [c["nx"], c["ny"], c["nz"]][:self.dim]
        self.h = 1.0 / max(self.cells)
        self.xmin = [0.0] * self.dim
        self.walls = (1 << (2 * self.dim)) - 1
        self.layers = 2
        self.gravity = [0.0] * self.dim
        self.gravity[-1] = -9.81
        self.rho, self.E, self.nu, self.K = 1e3, 1e6, 0.3, 2e6
        self.H = self.ty = 0.0
        if c["material"] == "vonmises":  # the copper rod of the Taylor impact
            self.R, self.L = 0.0032, 0.0324
            self.h = 6 * self.R / c["nx"]
            self.xmin = [-3 * self.R, -3 * self.R, 0.0]
            self.rho, self.E, self.nu, self.H, self.ty = 8.93e3, 117e9, 0.35, 0.1e9, 0.4e9
            self.walls, self.layers, self.gravity = 1 << 4, 1, [0.0] * 3
        if c["body"] == "disks":
            self.E, self.gravity = 500.0, [0.0] * self.dim
        if c["body"] == "clusters":
            self.E, self.nu = 1e5, 0.35
        self.lam = self.E * self.nu / ((1 + self.nu) * (1 - 2 * self.nu))
        self.mu = self.E / (2 * (1 + self.nu))
        if c["material"] == "fluid":
            self.mu, self.lam = 0.0, self.K
        self.V0 = (self.h / (2 if c["body"] == "clusters" else c["ppc"])) ** self.dim
        # a quarter of the acoustic time step; the clusters' crowded cells take less
        cs = math.sqrt((self.lam + 2 * self.mu) / self.rho)
        self.dt = (0.05 if c["body"] == "clusters" else 0.25) * self.h / cs
        self.gimp_l = self.h / c["ppc"]
        self.form = c["form"]
        self.T = F64 if self.form == "f64" else torch.float32
        self.xT = torch.float32 if self.form == "f32" else F64
        self.per_lame = c["body"] == "sphere"
        self.per_mass = c["body"] == "clusters"

    def extent(self):
        return [n * self.h for n in self.cells]

    def axis(self, d, lo, hi):
        """GridSampling points of axis d inside [lo, hi]."""
        l = self.h / self.c["ppc"]
        n = self.cells[d] * self.c["ppc"]
        a = self.xmin[d] + (2.0 * torch.arange(n, dtype=F64, device=DEV) + 1.0) * (l / 2)
        return a[(a >= lo) & (a <= hi)]

    def points(self, gen):
        """Particle positions (dim, n), first axis fastest."""
        c, D, X = self.c, self.dim, self.extent()
        lp = self.h / c["ppc"]
        if c["body"] == "clusters":
            n = c["count"]
            ctr = torch.stack([0.2 * X[d] + 0.6 * X[d] * torch.rand(64, dtype=F64, device=DEV, generator=gen)
                               for d in range(D)])
            which = torch.randint(0, 64, (n,), device=DEV, generator=gen)
            x = ctr[:, which] + 0.02 * min(X) * torch.randn(D, n, dtype=F64, device=DEV, generator=gen)
            for d in range(D):
                x[d].clamp_(0.02 * X[d], 0.98 * X[d])
            return x
        if c["body"] == "block":
            box = [(0.25 * X[d], 0.75 * X[d]) for d in range(D)]
        elif c["body"] == "column":
            box = [(0.0, 0.4 * X[0]), (0.0, X[1]), (0.0, 0.8 * X[2])]
        elif c["body"] == "rod":
            box = [(-self.R, self.R), (-self.R, self.R), (0.0, self.L)]
        else:
            box = [(0.0, X[d]) for d in range(D)]
        ax = [self.axis(d, *box[d]) for d in range(D)]
        g = torch.meshgrid(*reversed(ax), indexing="ij")
        x = torch.stack([t.reshape(-1) for t in reversed(g)])
        if c["body"] == "sphere":
            r = 0.3 * min(X)
            x = x[:, sum((x[d] - 0.5 * X[d]) ** 2 for d in range(D)) < r * r]
        elif c["body"] == "rod":
            x = x[:, x[0] ** 2 + x[1] ** 2 < self.R ** 2]
        elif c["body"] == "disks":
            r, m = 0.2 * min(X), min(X)
            a = sum((x[d] - 0.2 * m) ** 2 for d in range(D)) < r * r
            b = sum((x[d] - (X[d] - 0.2 * m)) ** 2 for d in range(D)) < r * r
            x = x[:, a | b]
        # on the lattice itself a uGIMP support ends at a node to the last bit
        if c["body"] in ("sphere", "rod", "column") or c["basis"].endswith("ugimp"):
            x = x + (torch.rand(x.shape, dtype=F64, device=DEV, generator=gen) - 0.5) * (lp / 2)
        return x.contiguous()

    def block_order(self, x):
        L = 2 if self.dim == 3 else 3
        b = torch.zeros(x.shape[1], dtype=torch.int64, device=x.device)
        for d in reversed(range(self.dim)):
            k = torch.floor((x[d] - self.xmin[d]) / self.h).long().clamp_(0, self.cells[d] - 1) >> L
            b = b * ((self.cells[d] >> L) + 1) + k
        return torch.argsort(b, stable=True)

    def inputs(self, seed):
        """The particle state in the precision form's types, from the seed alone."""
        c, D = self.c, self.dim
        gen = torch.Generator(device=DEV).manual_seed(int(seed))
        x = self.points(gen)
        if c["order"] == "block":
            x = x[:, self.block_order(x)].contiguous()
        x = x.to(self.xT)
        n = x.shape[1]
        # a smooth deformation: F = I + sum of plane waves
        waves = []
        for _ in range(3):
            k = torch.randn(D, dtype=F64, device=DEV, generator=gen) * (6.0 / max(self.extent()))
            waves.append((k, torch.randn(D, D, dtype=F64, device=DEV, generator=gen),
                          6.28 * torch.rand(1, dtype=F64, device=DEV, generator=gen)))
        amp = 2e-4 if c["material"] == "fluid" else 3e-3
        F = torch.zeros(D * D, n, dtype=F64, device=DEV)
        for k, A, ph in waves:
            s = torch.sin(sum(k[d] * x[d].double() for d in range(D)) + ph)
            if c["material"] == "vonmises":  # the foot of the rod is the deformed part
                s = 2.0 * s * torch.exp(-x[2].double() / self.R)
            for r in range(D):
                for q in range(D):
                    F[r + q * D].add_(s, alpha=float(amp * A[r, q]))
            del s
        for d in range(D):
            F[d + d * D] += 1.0
        u = {"x": x, "F": F}
        v = (torch.rand(D, n, dtype=F64, device=DEV, generator=gen) - 0.5)
        if c["material"] == "vonmises":
            v *= 2.0
            v[2] -= 227.0 * (1.0 - torch.exp(-x[2].double() / self.R))
        elif c["body"] == "disks":
            v *= 0.01
            v += torch.where(x[0].double() > 0.5 * self.extent()[0], -0.1, 0.1)
        elif c["material"] == "fluid":
            v *= 0.1
        u["v"] = v.to(self.T)
        del v
        if self.per_mass:
            z = torch.randn(n, dtype=F64, device=DEV, generator=gen)
            u["m"] = (self.rho * self.V0 * torch.exp(0.5 * z)).to(self.T)
        if self.per_lame:
            e = torch.exp(0.1 * torch.randn(n, dtype=F64, device=DEV, generator=gen))
            u["mu"], u["lam"] = (self.mu * e).to(self.T), (self.lam * e).to(self.T)
        mu, lam = (u["mu"].double(), u["lam"].double()) if self.per_lame else (self.mu, self.lam)
        J = det(F, D)
        if c["material"] == "fluid":
            sig = [lam * (J - 1.0) if i in diagonal(D) else torch.zeros_like(J) for i in range(nsym(D))]
        elif c["material"] == "vonmises":
            sig = hencky_guess(F, J, mu, lam, self.ty)
        else:
            sig = neo_hookean(F, J, mu, lam, D)
        u["sigma"] = torch.stack(sig).to(self.T)
        u["V"] = (self.V0 * J).to(self.T)
        if c["transfer"] == "apic":
            B = (torch.rand(D * D, n, dtype=F64, device=DEV, generator=gen) - 0.5)
            u["B"] = (B * (0.02 * self.h * (0.1 if c["material"] == "fluid" else 1.0))).to(self.T)
        if c["material"] == "vonmises":
            u["eps_p"] = torch.zeros(n, dtype=self.T, device=DEV)
            Cp = torch.zeros(6, n, dtype=self.T, device=DEV)
            Cp[0], Cp[3], Cp[5] = 1.0, 1.0, 1.0
            u["Cp_inv"] = Cp
        return u


def nsym(D):
    return 6 if D == 3 else 3


def diagonal(D):
    return (0, 3, 5) if D == 3 else (0, 2)


def sym(D, r, c):
    r, c = max(r, c), min(r, c)
    return c * D - c * (c - 1) // 2 + (r - c)


def det(F, D):
    f = lambda r, c: F[r + c * D]  # noqa: E731
    if D == 2:
        return f(0, 0) * f(1, 1) - f(0, 1) * f(1, 0)
    return (f(0, 0) * (f(1, 1) * f(2, 2) - f(1, 2) * f(2, 1)) - f(0, 1) * (f(1, 0) * f(2, 2) - f(1, 2) * f(2, 0))
            + f(0, 2) * (f(1, 0) * f(2, 1) - f(1, 1) * f(2, 0)))


def neo_hookean(F, J, mu, lam, D):
    """(mu (F F^T - I) + lambda log J I) / J, symmetric components."""
    lj = torch.log(J)
    out = [None] * nsym(D)
    for c in range(D):
        for r in range(c, D):
            b = sum(F[r + k * D] * F[c + k * D] for k in range(D))
            out[sym(D, r, c)] = (mu * (b - (1.0 if r == c else 0.0)) + (lam * lj if r == c else 0.0)) / J
    return out


def hencky_guess(F, J, mu, lam, ty):
    """A stress near the yield surface for the deformation F (small strains)."""
    kappa = lam + 2 * mu / 3
    e = [None] * 6
    for c in range(3):
        for r in range(c, 3):
            e[sym(3, r, c)] = 0.5 * (F[r + 3 * c] + F[c + 3 * r]) - (1.0 if r == c else 0.0)
    tr = (e[0] + e[3] + e[5]) / 3
    s = [2 * mu * (e[i] - (tr if i in diagonal(3) else 0.0)) for i in range(6)]
    q = torch.sqrt(1.5 * (s[0] ** 2 + s[3] ** 2 + s[5] ** 2 + 2 * (s[1] ** 2 + s[2] ** 2 + s[4] ** 2)))
    f = torch.clamp(ty / q.clamp_min(1.0), max=1.0)
    return [s[i] * f + (kappa * torch.log(J) / J if i in diagonal(3) else 0.0) for i in range(6)]


# --------------------------------------------------------------------------
# prepare, run
# --------------------------------------------------------------------------

class State:
    pass


def prepare(case, seed):
    tb = package()
    abi = tb._abi
    sc = Scene(case)
    s = State()
    s.rt = tb.runtime
    s.case, s.tb = case, tb
    s.mesh = tb.CartesianMesh(sc.h, *[(sc.xmin[d], sc.xmin[d] + sc.cells[d] * sc.h) for d in range(sc.dim)])
    basis = {"bspline": abi.TB_BSPLINE_QUADRATIC, "ugimp": abi.TB_UGIMP, "wls_bspline": abi.TB_WLS_BSPLINE_QUADRATIC,
             "wls_ugimp": abi.TB_WLS_UGIMP, "kc_bspline": abi.TB_KC_BSPLINE_QUADRATIC}[case["basis"]]
    material = {"neo": abi.MATERIAL_NEOHOOKEAN, "fluid": abi.MATERIAL_FLUID,
                "vonmises": abi.MATERIAL_VONMISES}[case["material"]]
    s.params = tb.step_params(sc.dt, mass=sc.rho * sc.V0, V0=sc.V0, mu=sc.mu, lam=sc.lam, gravity=sc.gravity,
                              gimp_l=sc.gimp_l, flip_alpha=case["alpha"], basis=basis,
                              transfer=abi.TB_TRANSFER_APIC if case["transfer"] == "apic" else abi.TB_TRANSFER_FLIP,
                              material=material, wall_mask=sc.walls, wall_layers=sc.layers, hardening=sc.H,
                              yield_stress=sc.ty)
    u = sc.inputs(seed)
    n = u["x"].shape[1]
    opt = tuple(k for k in ("m", "mu", "lam", "B", "eps_p", "Cp_inv") if k in u)
    host = case["kind"] == "host"
    P = tb.Particles(n, sc.dim, "float64" if sc.form == "f64" else "float32", "pinned" if host else "torch",
                     None if host else DEV, optional=opt, x64=sc.form == "f32x64")
    for k, t in u.items():
        if host:
            getattr(P, k)[...] = t.cpu().numpy()
        else:
            getattr(P, k).copy_(t)
    s.particles = P
    if case["kind"] in ("step", "loop", "adaptive"):
        s.grid = tb.generate_grid(s.mesh, P.dtype, backend="torch", device=DEV)
        s.part = tb.Partition(s.mesh, n, backend="torch", device=DEV)
    if case["kind"] == "grad":
        s.target = [0.5 * e for e in sc.extent()]
        s.target[-1] = 0.8 * sc.extent()[-1]
    return s


def loss_and_grad(target):
    """Mean squared distance of the particles to a target point, and its gradient."""
    def f(P):
        d = P.x.double() - torch.tensor(target, dtype=F64, device=P.x.device)[:, None]
        return (d * d).sum() / P.n, d * (2.0 / P.n), torch.zeros_like(d)
    return f


def run(s):
    rt, c, P = s.rt, s.case, s.particles
    if c["kind"] == "grad":
        loss, gv, ge = rt.rollout_grad(P, s.mesh, s.params, c["steps"], loss_and_grad(s.target))
        return {"loss": loss, "dv0": gv, **({} if ge is None else {"dlogE": ge})}
    if c["kind"] == "host":
        rt.rollout_host(P, s.mesh, s.params, c["steps"])
        return state_of(P)
    t = None
    if c["kind"] == "step":
        rt.step(s.grid, P, s.part, s.mesh, s.params, c["steps"])
    elif c["kind"] == "adaptive":
        t = rt.adaptive_steps(s.grid, P, s.part, s.mesh, s.params, c["steps"])
    else:
        rt.update(s.part, P, s.mesh)
        rt.P2G(s.grid, P, s.part, s.mesh, s.params)
        rt.G2P(s.grid, P, s.mesh, s.params)
    g = s.grid
    # not grid.v and grid.vn: at nodes that a window only touches they are the
    # ratio of two sums near zero, which no two orders of summation share; the
    # particles' v and grad_v carry them with their weights
    out = {**state_of(P), "grid_m": g.m, "grid_mv": g.mv, "grid_f": g.f}
    if t is not None:
        out["time"] = t
    if c["kind"] == "loop":
        out["order"] = s.part.particleindices
    return out


def state_of(P):
    return {k: getattr(P, k) for k in ("x", "v", "V", "grad_v", "sigma", "F", "B", "eps_p", "Cp_inv")
            if getattr(P, k) is not None}


# --------------------------------------------------------------------------
# work
# --------------------------------------------------------------------------

def work(case):
    """Bytes and operations of one pass: per step each particle field the step
    reads and writes once, per call every node of the grid arrays written once
    (a dense grid's nodes are all outputs), per further step the body's nodes."""
    sc = Scene(case)
    D, T = sc.dim, 8 if sc.form == "f64" else 4
    xb = 4 if sc.form == "f32" else 8
    X = sc.extent()
    vol = {"block": 0.5 ** D * math.prod(X), "column": 0.32 * math.prod(X),
           "sphere": 4 / 3 * math.pi * (0.3 * min(X)) ** 3, "disks": 2 * math.pi * (0.2 * min(X)) ** 2}
    if case["body"] == "clusters":
        n = case["count"]
        nodes = min(n, 0.05 * math.prod(sc.cells))
    elif case["body"] == "rod":
        cells = math.pi * sc.R ** 2 * sc.L / sc.h ** 3
        n, nodes = cells * 27, cells * 1.3
    else:
        cells = vol[case["body"]] / sc.h ** D
        n, nodes = cells * case["ppc"] ** D, cells * 1.1
    apic = case["transfer"] == "apic"
    rd = D * xb + (D + 1 + nsym(D)) * T + D * D * 8 + (D * D * T if apic else 0)
    rd += (T if sc.per_mass else 0) + (2 * T if sc.per_lame else 0)
    wr = D * xb + (D + 1 + nsym(D) + D * D) * T + D * D * 8 + (D * D * T if apic else 0)
    if case["material"] == "vonmises":
        rd += 7 * T
        wr += 7 * T
    nn = math.prod(k + 1 for k in sc.cells)
    per_node = (1 + 4 * D) * T
    flops = n * 3 ** D * (2 * (1 + 2 * D) + 2 * (2 * D + D * D) + (60 if case["basis"].startswith("wls") else 20))
    k = case["steps"]
    if case["kind"] == "grad":
        # forward steps keep their state; the reverse steps read it, and read and
        # write the FP64 sensitivities of x, v, F (B)
        adj = 8 * (2 * D + D * D + (D * D if apic else 0))
        b = k * (n * (rd + wr + (rd + 2 * adj)) + 2 * nodes * per_node)
        return {"bytes": float(b), "flops": float(k * flops * 4)}
    calls = k if case["kind"] == "adaptive" else 1
    b = k * n * (rd + wr) + calls * nn * per_node + (k - calls) * nodes * per_node
    return {"bytes": float(b), "flops": float(k * flops)}


# --------------------------------------------------------------------------
# the step in plain torch, FP64
# --------------------------------------------------------------------------

def jet_bspline(xi):
    a, s = xi.abs(), torch.sign(xi)
    val = torch.where(a < 0.5, 0.75 - a * a, torch.where(a < 1.5, 0.5 * (1.5 - a) ** 2, torch.zeros_like(a)))
    der = torch.where(a < 0.5, -2 * a, torch.where(a < 1.5, -(1.5 - a), torch.zeros_like(a))) * s
    return val, der


def jet_ugimp(xi, l):
    a, s = xi.abs(), torch.sign(xi)
    z = torch.zeros_like(a)
    t = 1 + l / 2 - a
    val = torch.where(a < l / 2, 1 - (4 * a * a + l * l) / (4 * l),
                      torch.where(a < 1 - l / 2, 1 - a, torch.where(a < 1 + l / 2, t * t / (2 * l), z)))
    der = torch.where(a < l / 2, -2 * a / l, torch.where(a < 1 - l / 2, -torch.ones_like(a),
                                                         torch.where(a < 1 + l / 2, -t / l, z))) * s
    return val, der


class Weights:
    """Nodes, weights and gradients of the particles at x (D, n)."""

    def __init__(self, sc, x):
        D, h, name = sc.dim, sc.h, sc.c["basis"]
        gimp = name.endswith("ugimp")
        l = sc.gimp_l / h
        self.D, self.wls, self.apic_r = D, name.startswith("wls"), None
        self.node, self.val, self.der, self.rel = [], [], [], []
        cut = torch.zeros(x.shape[1], dtype=torch.bool, device=x.device)
        full = []
        for d in range(D):
            xi = (x[d] - sc.xmin[d]) / h
            with torch.no_grad():
                lo = (torch.floor(xi - (1 + l / 2)) + 1 if gimp else torch.floor(xi - 0.5)).long()
            N, V, G, R, inside = [], [], [], [], []
            for k in range(3):
                i = lo + k
                ok = (i >= 0) & (i < sc.cells[d] + 1)
                r = (sc.xmin[d] + i.double() * h) - x[d]
                val, der = jet_ugimp(-r / h, l) if gimp else jet_bspline(-r / h)
                z = torch.zeros_like(val)
                N.append(i.clamp(0, sc.cells[d]))
                V.append(torch.where(ok, val, z))
                G.append(torch.where(ok, der / h, z))
                R.append(r)
                inside.append(ok)
            f = inside[0] & inside[1] & inside[2]
            full.append(f)
            cut |= ~f
            self.node.append(N)
            self.val.append(V)
            self.der.append(G)
            self.rel.append(R)
        if name.startswith("kc"):
            # 1-D fits on the supports that the mesh cuts
            for d in range(D):
                S = [sum(self.val[d][k] * self.rel[d][k] ** p for k in range(3)) for p in range(3)]
                den = S[0] * S[2] - S[1] * S[1]
                for k in range(3):
                    w, r = self.val[d][k], self.rel[d][k]
                    fit = w * (S[2] - S[1] * r) / den
                    fit_d = torch.where(full[d], w * r * (4 / h ** 2), w * (S[0] * r - S[1]) / den)
                    self.val[d][k] = torch.where(cut & ~full[d], fit, w)
                    self.der[d][k] = torch.where(cut, fit_d, self.der[d][k])
        if self.wls:
            S = [[sum(self.val[d][k] * self.rel[d][k] ** p for k in range(3)) for p in range(3)] for d in range(D)]
            M = torch.empty(x.shape[1], D + 1, D + 1, dtype=F64, device=x.device)
            for a in range(D + 1):
                rows = []
                for b in range(D + 1):
                    t = 1.0
                    for d in range(D):
                        t = t * S[d][(a == d + 1) + (b == d + 1)] / h ** ((a == d + 1) + (b == d + 1))
                    rows.append(t)
                M = M.clone() if M.requires_grad else M
                M[:, a] = torch.stack(rows, dim=-1)
            self.Mi = torch.linalg.inv(M)  # of the moments of (1, r / h)
            self.h = h

    def at(self, i, j, k):
        """w, grad w and X - x at window slot (i, j, k)."""
        ijk, D = (i, j, k), self.D
        v = [self.val[d][ijk[d]] for d in range(D)]
        w = math.prod(v[1:], start=v[0])
        r = [self.rel[d][ijk[d]] for d in range(D)]
        if self.wls:
            p = [1.0] + [t / self.h for t in r]
            q = [w * sum(self.Mi[:, a, b] * p[b] for b in range(D + 1)) for a in range(D + 1)]
            return q[0], [t / self.h for t in q[1:]], r
        g = []
        for a in range(D):
            t = self.der[a][ijk[a]]
            for d in range(D):
                if d != a:
                    t = t * v[d]
            g.append(t)
        return w, g, r

    def slots(self):
        return [(i, j, k) for k in range(3 if self.D == 3 else 1) for j in range(3) for i in range(3)]

    def nodes(self, sc, i, j, k):
        n = self.node[0][i] + (sc.cells[0] + 1) * self.node[1][j]
        return n if self.D == 2 else n + (sc.cells[0] + 1) * (sc.cells[1] + 1) * self.node[2][k]


def p2g_exact(sc, u, lo, hi, W, grid):
    """Adds the particles lo..hi to the sums grid = (m, mv, f)."""
    D, h = sc.dim, sc.h
    cut = lambda t: t[..., lo:hi]  # noqa: E731
    m = cut(u["m"]) if sc.per_mass else torch.full((hi - lo,), sc.rho * sc.V0, dtype=F64, device=DEV)
    v, V = cut(u["v"]), cut(u["V"])
    s = [cut(t) for t in u["sigma"]]
    B = cut(u["B"]) if "B" in u else None
    gm, gmv, gf = grid
    for i, j, k in W.slots():
        w, g, r = W.at(i, j, k)
        at = W.nodes(sc, i, j, k)
        gm = gm.index_add(0, at, w * m) if gm.requires_grad or w.requires_grad else gm.index_add_(0, at, w * m)
        for a in range(D):
            va = v[a]
            if B is not None:
                va = va + sum(B[a + c * D] * r[c] for c in range(D)) * (4 / h ** 2)
            fa = -V * sum(s[sym(D, a, c)] * g[c] for c in range(D)) + w * m * sc.gravity[a]
            if fa.requires_grad or gmv[a].requires_grad:
                gmv[a], gf[a] = gmv[a].index_add(0, at, w * m * va), gf[a].index_add(0, at, fa)
            else:
                gmv[a].index_add_(0, at, w * m * va)
                gf[a].index_add_(0, at, fa)
    return gm, gmv, gf


def grid_exact(sc, gm, gmv, gf, dt):
    on = gm != 0
    ms = torch.where(on, gm, torch.ones_like(gm))
    z = torch.zeros_like(gm)
    vn = [torch.where(on, t / ms, z) for t in gmv]
    v = [torch.where(on, vn[d] + dt * gf[d] / ms, z) for d in range(sc.dim)]
    idx = torch.arange(gm.shape[0], device=DEV)
    for d in range(sc.dim):
        i = idx % (sc.cells[d] + 1)
        idx = idx // (sc.cells[d] + 1)
        wall = torch.zeros_like(on)
        if (sc.walls >> (2 * d)) & 1:
            wall |= i < sc.layers
        if (sc.walls >> (2 * d + 1)) & 1:
            wall |= i >= sc.cells[d] + 1 - sc.layers
        vn[d], v[d] = torch.where(wall, z, vn[d]), torch.where(wall, z, v[d])
    return vn, v


def g2p_exact(sc, u, lo, hi, W, vn, v, dt, mu, lam):
    D, c = sc.dim, sc.c
    cut = lambda t: t[..., lo:hi]  # noqa: E731
    z = torch.zeros(hi - lo, dtype=F64, device=DEV)
    pic, dv = [z] * D, [z] * D
    gv = [z] * (D * D)
    Bn = [z] * (D * D)
    for i, j, k in W.slots():
        w, g, r = W.at(i, j, k)
        at = W.nodes(sc, i, j, k)
        for a in range(D):
            va = v[a][at]
            wv = w * va
            pic[a] = pic[a] + wv
            dv[a] = dv[a] + (wv - w * vn[a][at])
            for q in range(D):
                gv[a + q * D] = gv[a + q * D] + va * g[q]
                if "B" in u:
                    Bn[a + q * D] = Bn[a + q * D] + wv * r[q]
    o = {"x": torch.stack([cut(u["x"])[d] + pic[d] * dt for d in range(D)])}
    if c["transfer"] == "apic":
        o["v"], o["B"] = torch.stack(pic), torch.stack(Bn)
    else:
        a = c["alpha"]
        o["v"] = torch.stack([(1 - a) * pic[d] + a * (cut(u["v"])[d] + dv[d]) for d in range(D)])
    o["grad_v"] = torch.stack(gv)
    A = [gv[r + q * D] * dt + (1.0 if r == q else 0.0) for q in range(D) for r in range(D)]
    F0 = cut(u["F"])
    F = [sum(A[r + k * D] * F0[k + q * D] for k in range(D)) for q in range(D) for r in range(D)]
    o["F"] = torch.stack(F)
    J = det(F, D)
    mu, lam = (cut(mu), cut(lam)) if torch.is_tensor(mu) else (mu, lam)
    if c["material"] == "vonmises":
        o.update(vonmises_exact(sc, F, J, det(A, 3), mu, lam, cut(u["V"]), cut(u["eps_p"]), cut(u["Cp_inv"])))
        return o
    if c["material"] == "fluid":
        sig = [lam * (J - 1.0) if i in diagonal(D) else z for i in range(nsym(D))]
    else:
        sig = neo_hookean(F, J, mu, lam, D)
    o["sigma"], o["V"] = torch.stack(sig), sc.V0 * J
    return o


def vonmises_exact(sc, F, J, dJ, mu, lam, V, ep, Cp):
    n = J.shape[0]
    M = lambda f: torch.stack([torch.stack([f(r, q) for q in range(3)], -1) for r in range(3)], -2)  # noqa: E731
    Fm = M(lambda r, q: F[r + 3 * q])
    C = M(lambda r, q: Cp[sym(3, r, q)])
    b = Fm @ C @ Fm.transpose(1, 2)
    b = 0.5 * (b + b.transpose(1, 2))
    ev, nv = torch.empty(n, 3, dtype=F64, device=DEV), torch.empty(n, 3, 3, dtype=F64, device=DEV)
    for a in range(0, n, 16384):
        ev[a:a + 16384], nv[a:a + 16384] = torch.linalg.eigh(b[a:a + 16384])
    lj = torch.log(J)[:, None]
    le = 0.5 * torch.log(ev)
    tau = 2 * mu * le - 2 * mu / 3 * lj
    nrm = torch.sqrt(1.5 * (tau * tau).sum(1, keepdim=True))
    f = nrm - (sc.ty + sc.H * ep[:, None])
    dg = torch.where(f > 0, f / (3 * mu + sc.H), torch.zeros_like(f))
    de = dg * 1.5 * tau / nrm.clamp_min(1e-300)
    le = le - de
    tau = tau - 2 * mu * de
    pr = ((lam + 2 * mu / 3) * lj / J[:, None])
    s = (nv * (tau / J[:, None] + pr)[:, None, :]) @ nv.transpose(1, 2)
    m = torch.linalg.inv(Fm) @ nv
    Ci = (m * torch.exp(2 * le)[:, None, :]) @ m.transpose(1, 2)
    pick = lambda t: torch.stack([t[:, r, q] for q in range(3) for r in range(q, 3)])  # noqa: E731
    return {"sigma": pick(s), "Cp_inv": pick(Ci), "eps_p": ep + dg[:, 0], "V": dJ * V}


def step_exact(sc, u, dt, mu, lam, chunk=1 << 21):
    n, N = u["x"].shape[1], math.prod(k + 1 for k in sc.cells)
    zero = lambda: torch.zeros(N, dtype=F64, device=DEV)  # noqa: E731
    grid = (zero(), [zero() for _ in range(sc.dim)], [zero() for _ in range(sc.dim)])
    for lo in range(0, n, chunk):
        hi = min(n, lo + chunk)
        grid = p2g_exact(sc, u, lo, hi, Weights(sc, u["x"][:, lo:hi]), grid)
    vn, v = grid_exact(sc, *grid, dt)
    parts = []
    for lo in range(0, n, chunk):
        hi = min(n, lo + chunk)
        parts.append(g2p_exact(sc, u, lo, hi, Weights(sc, u["x"][:, lo:hi]), vn, v, dt, mu, lam))
    o = dict(u)
    for k in parts[0]:
        o[k] = torch.cat([p[k] for p in parts], dim=-1) if len(parts) > 1 else parts[0][k]
    return o, grid


def exact(case, seed):
    sc = Scene(case)
    u = {k: t.double() for k, t in sc.inputs(seed).items()}
    mu, lam = (u["mu"], u["lam"]) if sc.per_lame else (sc.mu, sc.lam)
    if case["kind"] == "grad":
        return grad_exact(sc, u, mu, lam)
    t = 0.0
    with torch.no_grad():
        for _ in range(case["steps"]):
            dt = sc.dt
            if case["kind"] == "adaptive":
                cs = torch.sqrt((lam + 2 * mu) * u["V"] / (sc.rho * sc.V0)) + torch.sqrt((u["v"] ** 2).sum(0))
                dt = 0.8 * sc.h / float(cs.max())
            u, grid = step_exact(sc, u, dt, mu, lam)
            t += dt
    out = {k: u[k] for k in ("x", "v", "V", "grad_v", "sigma", "F", "B", "eps_p", "Cp_inv") if k in u}
    if case["kind"] == "host":
        return out
    out.update(grid_m=grid[0], grid_mv=torch.stack(grid[1]), grid_f=torch.stack(grid[2]))
    if case["kind"] == "adaptive":
        out["time"] = t
    if case["kind"] == "loop":
        out["order"] = None
    return out


def grad_exact(sc, u, mu, lam):
    """Reverse-mode derivatives of the torch steps, recomputed step by step."""
    D, keys = sc.dim, [k for k in ("x", "v", "F", "B") if k in u]
    with torch.enable_grad():
        v0 = u["v"].clone().requires_grad_(True)
        s = torch.zeros(u["x"].shape[1], dtype=F64, device=DEV, requires_grad=True) if sc.per_lame else None
        mu_s, lam_s = (mu * torch.exp(s), lam * torch.exp(s)) if sc.per_lame else (mu, lam)

        def one(*a):
            w = dict(zip(keys, a))
            if sc.per_lame:
                w_mu, w_lam = a[len(keys)], a[len(keys) + 1]
            else:
                w_mu, w_lam = mu, lam
            J = det(w["F"], D)
            if sc.c["material"] == "fluid":
                sig = [w_lam * (J - 1.0) if i in diagonal(D) else torch.zeros_like(J) for i in range(nsym(D))]
            else:
                sig = neo_hookean(w["F"], J, w_mu, w_lam, D)
            w["sigma"], w["V"] = torch.stack(sig), sc.V0 * J
            o, _ = step_exact(sc, w, sc.dt, w_mu, w_lam, chunk=1 << 40)
            return tuple(o[k] for k in keys)

        a = tuple(v0 if k == "v" else u[k] for k in keys)
        for _ in range(sc.c["steps"]):
            extra = (mu_s, lam_s) if sc.per_lame else ()
            a = torch.utils.checkpoint.checkpoint(one, *a, *extra, use_reentrant=False)
        target = [0.5 * e for e in sc.extent()]
        target[-1] = 0.8 * sc.extent()[-1]
        d = a[0] - torch.tensor(target, dtype=F64, device=DEV)[:, None]
        loss = (d * d).sum() / d.shape[1]
        loss.backward()
    return {"loss": loss.detach(), "dv0": v0.grad, **({"dlogE": s.grad} if sc.per_lame else {})}
