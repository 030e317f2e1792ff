"""What this framework is timed on: whole simulations through its public API.

A pass is what a program has the library do for one scene (or one batch of
scenes): construct the solver from particles in pinned host memory, advance it,
and read the state back into pinned host memory.  Every pass starts from the
same particles, so passes repeat exactly.  Forms:

  solve    MPMSolver3D / APICMPMSolver3D, steps, read-back
  batch    many scenes of uneven size in one Batch
  export   steps, then the density grid that writeToOpenVDB rasterises
  objects  CFL time step, level-set collision object, particle collision
  implicit the semi-implicit update (a conjugate-residual solve every step)

Step counts are a few frames' worth: beyond some tens of steps two roundings of
the same simulation drift apart in 32 bits (light nodes at a body's surface).
"""
import math

import numpy as np
import torch

from mpm_b200 import _abi
from mpm_b200.batch import Batch
from mpm_b200.level_set import LevelSetCollisionObject3D, sphere
from mpm_b200.scenes import Scene
from mpm_b200.solver import Material, Particles

SNOW = dict(youngs_modulus=1.4e5, poisson_ratio=0.2, hardening=10.0, critical_compression=2.5e-2,
            critical_stretch=7.5e-3)
DENSITY = 400.0
FLT_EPS = float(np.finfo(np.float32).eps)
SPLINE = {"linear": _abi.INTERP_LINEAR, "quadratic": _abi.INTERP_QUADRATIC, "cubic": _abi.INTERP_CUBIC}
NODES = {"linear": 2, "quadratic": 3, "cubic": 4}
FIELDS = {"position": (_abi.FIELD_POSITION, 3), "velocity": (_abi.FIELD_VELOCITY, 3),
          "det_fe": (_abi.FIELD_DET_FE, 1)}


def _case(form, shape, n, res, spline, apic, steps, **more):
    """A case: `n` particles of `shape` on a res^3 grid of the unit cube; dt is
    dt_cells times the cell size (0.0064 in the benchmark configurations)."""
    c = dict(form=form, shape=shape, n=n, res=res, spline=spline, apic=apic, steps=steps, extent=0.3, speed=2.0,
             dt_cells=0.0064, sticky=True, materials=1, neo_hookean=False)
    c.update(more)
    return c


def listed():
    cases = {
        # a unit test's or an interactive demo's scene, reference boundary: launches and latency only
        "demo_4k_cubic_apic": _case("solve", "box", 4096, 24, "cubic", True, 30, sticky=False),
        # the plain configuration: the snow cube of 65,536 particles, quadratic PIC-FLIP
        "snow_cube_65k_quadratic_flip": _case("solve", "box", 65536, 64, "quadratic", False, 40),
        # the reference's two-material ball collision (63,008 particles, 200^3, cubic PIC-FLIP), denser in its cells
        "two_materials_63k_cubic_flip": _case("solve", "balls", 63008, 200, "cubic", False, 30, extent=0.11,
                                              speed=2.5, sticky=False, materials=2),
        # the cheapest kernel of the reference on a ragged count, with its other constitutive model
        "linear_200k_neo_hookean": _case("solve", "sphere", 200_003, 96, "linear", False, 12, extent=0.4,
                                         neo_hookean=True),
        # two balls of half a million particles each, cubic APIC on 128^3
        "two_balls_1m_cubic_apic": _case("solve", "balls", 1_048_576, 128, "cubic", True, 30, extent=0.24, speed=3.0),
        # the largest request of the serving stream: 2M particles, many per cell
        "request_2m_quadratic_apic": _case("solve", "box", 2_000_000, 128, "quadratic", True, 25, speed=3.1),
        # the large scene: slab and falling sphere, 8,388,608 particles, about 3 per cell of a 256^3 grid
        "slab_8m_cubic_apic": _case("solve", "slab", 8_388_608, 256, "cubic", True, 12, speed=5.0),
        # 64 independent scenes of 10k to 500k particles, half APIC and half PIC-FLIP, as one batch
        "batch_64_quadratic_mixed": _case("batch", "mixed", 500_000, 128, "quadratic", True, 16, n_min=10_000,
                                          scenes=64),
        # a serving loop's usual moment: a few small scenes in flight
        "batch_6_small": _case("batch", "mixed", 60_000, 64, "quadratic", True, 30, n_min=5_000, scenes=6),
        # an offline frame: steps, then the density grid for the renderer
        "export_300k_density": _case("export", "sphere", 300_000, 128, "quadratic", True, 10, extent=0.35),
        # the collision features together: CFL step, level-set object, particle collision
        "objects_131k_cubic_apic": _case("objects", "box", 131_072, 64, "cubic", True, 24, speed=4.0, cfl=0.2),
        # backward Euler at ten times the explicit step
        "implicit_120k_cubic_apic": _case("implicit", "box", 120_000, 64, "cubic", True, 3, dt_cells=0.064,
                                          beta=1.0),
    }
    return [dict(c, name=k) for k, c in cases.items()]


def draw(rng):
    """One more case: a form, a stencil, a transfer, a particle count (log-uniform from a few hundred to 4M), particles
    per cell from the sparse slab's to the serving stream's, and the grid that these give."""
    form = rng.choice(["solve"] * 5 + ["batch"] * 2 + ["export", "objects", "implicit"])
    spline, apic = rng.choice([("linear", False), ("quadratic", False), ("quadratic", True), ("cubic", False),
                               ("cubic", True), ("cubic", True)])
    top = {"solve": 4e6, "batch": 2e5, "export": 1e6, "objects": 1e6, "implicit": 2e5}[form]
    n = int(math.exp(rng.uniform(math.log(600.0), math.log(top))))
    if form == "batch":
        return _case("batch", "mixed", max(n, 5000), rng.choice([64, 96, 128]), "quadratic", True,
                     rng.randint(8, 30), n_min=2000, scenes=rng.randint(2, 40))
    per_cell = math.exp(rng.uniform(math.log(2.5), math.log(32.0)))
    extent = rng.uniform(0.15, 0.5)
    res = int(min(256, max(16, round((n / per_cell) ** (1.0 / 3.0) / extent))))
    work = n * NODES[spline] ** 3 * (12 if form == "implicit" else 1)
    steps = int(min(rng.randint(8, 12 if spline == "linear" else 30), max(4, 3e9 // work)))
    more = {"cfl": 0.2} if form == "objects" else {"beta": rng.choice([0.5, 1.0]), "dt_cells": 0.05} \
        if form == "implicit" else {}
    if form == "implicit":
        steps = min(steps, 4)
    return _case(form, rng.choice(["box", "sphere", "balls"]), n, res, spline, apic, steps, extent=extent,
                 speed=rng.uniform(0.5, 5.0), sticky=rng.random() < 0.6, materials=rng.choice([1, 1, 2]),
                 neo_hookean=rng.random() < 0.2, **more)


# ---- inputs -----------------------------------------------------------------

def _ball(rng, n, center, radius):
    """n points uniform in a ball: a direction and a radius of density r^2."""
    d = rng.standard_normal((n, 3), dtype=np.float32)
    d *= (radius * np.cbrt(rng.random(n, dtype=np.float32)) / np.maximum(np.linalg.norm(d, axis=1), 1e-12))[:, None]
    return d + np.asarray(center, np.float32)


def _pinned(a):
    t = torch.empty(a.shape, dtype=getattr(torch, str(a.dtype)), pin_memory=torch.cuda.is_available())
    t.numpy()[...] = a
    return t.numpy()


def _scene(case, rng, shape, n, res, apic, steps, materials):
    e, s = case["extent"], np.float32(case["speed"])
    v = np.zeros((n, 3), np.float32)
    mat = None
    if shape == "slab":
        lo, hi, r = np.array([0.1, 0.05, 0.1]), np.array([0.9, 0.3, 0.9]), 0.1
        slab, ball = float(np.prod(hi - lo)), 4 / 3 * math.pi * r ** 3
        k, vol = n - int(round(n * ball / (slab + ball))), slab + ball
        x = np.concatenate([(lo + (hi - lo) * rng.random((k, 3), dtype=np.float32)).astype(np.float32),
                            _ball(rng, n - k, (0.5, 0.7, 0.5), r)])
        v[k:, 1] = -s
    elif shape == "balls":
        r, k = min(e / 2, 0.18), n // 2
        x = np.concatenate([_ball(rng, k, (0.3, 0.5, 0.5), r), _ball(rng, n - k, (0.7, 0.5, 0.5), r)])
        v[:k, 0], v[k:, 0], vol = s, -s, 2 * 4 / 3 * math.pi * r ** 3
        mat = (np.arange(n) >= k).astype(np.uint16)
    else:
        c = rng.uniform(0.2 + e / 2, 0.8 - e / 2, 3) if case["form"] == "batch" else np.array([0.5, 0.5, 0.5])
        d = rng.normal(size=3) + (0.0, -2.0, 0.0)
        v[:] = s * (d / np.linalg.norm(d)).astype(np.float32)
        if shape == "sphere":
            x, vol = _ball(rng, n, c, e / 2), 4 / 3 * math.pi * (e / 2) ** 3
        else:
            x, vol = rng.random((n, 3), dtype=np.float32) * np.float32(e) + (c - e / 2).astype(np.float32), e ** 3
        mat = (x[:, 1] > c[1]).astype(np.uint16)
    model = _abi.MODEL_NEO_HOOKEAN if case["neo_hookean"] else _abi.MODEL_FIXED_COROTATED
    mats = [Material(model=model, **dict(SNOW, **materials))]
    if case["materials"] == 2:
        mats.append(Material(model=model, **dict(SNOW, **materials, critical_compression=5e-2,
                                                 critical_stretch=9e-3)))
    m = np.full(n, DENSITY * vol / n, np.float32)
    p = Particles(_pinned(x), _pinned(v), _pinned(m), mats, _pinned(mat) if len(mats) > 1 else None)
    h = 1.0 / res
    return Scene("case", p, (0.0, 0.0, 0.0), (res, res, res), h, case["dt_cells"] * h,
                 _abi.TRANSFER_APIC if apic else _abi.TRANSFER_PIC_FLIP, SPLINE[case["spline"]], steps=steps,
                 boundary=_abi.BOUNDARY_STICKY if case["sticky"] else _abi.BOUNDARY_REFERENCE)


def _scenes(case, seed):
    """The scenes of a case.  A batch's sizes, grids and speeds are the case's own (every seed costs the same); its
    positions and materials come from the seed."""
    if case["form"] != "batch":
        rng = np.random.default_rng(np.random.SeedSequence([seed, 1]))
        return [_scene(case, rng, case["shape"], case["n"], case["res"], case["apic"], case["steps"], {})]
    sizes = np.random.default_rng(np.random.SeedSequence([17, case["n"], case["scenes"]]))
    out = []
    for i in range(case["scenes"]):
        n = int(round(math.exp(sizes.uniform(math.log(case["n_min"]), math.log(case["n"])))))
        res = int(sizes.choice([r for r in (32, 64, 96, 128) if r <= case["res"]]))
        one = dict(case, extent=float(sizes.uniform(0.1, 0.3)), speed=float(sizes.uniform(0.0, 4.0)))
        shape = "box" if sizes.random() < 0.5 else "sphere"
        rng = np.random.default_rng(np.random.SeedSequence([seed, i]))
        material = dict(youngs_modulus=rng.uniform(5e4, 2e5), hardening=rng.uniform(5, 10),
                        critical_compression=rng.uniform(1.5e-2, 3e-2), critical_stretch=rng.uniform(5e-3, 1e-2))
        out.append(_scene(one, rng, shape, n, res, i % 2 == 0, case["steps"], material))
    return out


def _object(sc):
    """A sphere under the body that it falls on, at rest."""
    return LevelSetCollisionObject3D(sphere(sc.origin, sc.resolution, sc.stride, (0.5, 0.22, 0.5), 0.16), 0.4)


def prepare(case, seed):
    scenes = _scenes(case, seed)
    total = sum(s.n for s in scenes)
    out = {k: torch.empty((total, c) if c > 1 else (total,), pin_memory=torch.cuda.is_available())
           for k, (_, c) in FIELDS.items()}
    return {"case": case, "scenes": scenes, "out": out,
            "object": _object(scenes[0]) if case["form"] == "objects" else None}


def run(state):
    case, scenes, out = state["case"], state["scenes"], state["out"]
    if case["form"] == "batch":
        with Batch() as b:
            ids = [b.add(s) for s in scenes]
            b.step(case["steps"])
            first = 0
            for sid, s in zip(ids, scenes):
                for name, (field, comps) in FIELDS.items():
                    b.download_async(sid, field, out[name].data_ptr() + 4 * comps * first)
                first += s.n
            b.download_wait()
        return out
    with scenes[0].solver() as g:
        if case["form"] == "objects":
            g.set_cfl(case["cfl"])
            g.set_collision_object(state["object"])
            g.switchIfEnableParticlesCollision()
        elif case["form"] == "implicit":
            g.set_implicit(case["beta"], max_iter=60, tol=1e-6)
        g.step(case["steps"])
        for name, (field, _) in FIELDS.items():
            g.download_async(field, out[name].data_ptr())
        got = dict(out)
        if case["form"] == "export":
            got["density"] = g.density()
        g.download_wait()
    return got


def work(case):
    """Bytes: the particles in, the state read and written once a step (200 B a particle in PIC-FLIP, 272 B in APIC),
    the fields out; the nodes of the scene's volume with the fields of one step (104 and 56 B).  Operations: the
    transfers' multiplies and adds per stencil node and the particle update's."""
    total = {"bytes": 0.0, "flops": 0.0}
    if case["form"] == "batch":
        sizes = np.random.default_rng(np.random.SeedSequence([17, case["n"], case["scenes"]]))
        parts = []
        for i in range(case["scenes"]):
            n = int(round(math.exp(sizes.uniform(math.log(case["n_min"]), math.log(case["n"])))))
            res = int(sizes.choice([r for r in (32, 64, 96, 128) if r <= case["res"]]))
            e = float(sizes.uniform(0.1, 0.3))
            sizes.uniform(0.0, 4.0)
            vol = e ** 3 if sizes.random() < 0.5 else math.pi / 6 * e ** 3
            parts.append((n, res, vol, i % 2 == 0))
    else:
        e = case["extent"]
        vol = {"box": e ** 3, "sphere": math.pi / 6 * e ** 3, "slab": 0.1642,
               "balls": math.pi / 3 * min(e, 0.36) ** 3}[case["shape"]]
        parts = [(case["n"], case["res"], vol, case["apic"])]
    for n, res, vol, apic in parts:
        nodes, steps, S3 = vol * res ** 3, case["steps"], NODES[case["spline"]] ** 3
        total["bytes"] += n * 56.0 + steps * (n * (272.0 if apic else 200.0) + nodes * (56.0 if apic else 104.0))
        flops = S3 * (44.0 if apic else 40.0) + 700.0
        if case["form"] == "implicit":  # a gather and a scatter of 3 components by 3 derivatives an iteration, ~5
            flops += 6 * (S3 * 36.0 + 300.0)
        total["flops"] += steps * n * flops
        if case["form"] == "export":
            total["bytes"] += 4.0 * res ** 3
    return total


# ---- the same steps in 64 bits ----------------------------------------------

def _spline(name, d):
    t = d.abs()
    if name == "linear":
        return (1 - t).clamp(min=0), torch.where((t < 1) & (t > FLT_EPS), -torch.sign(d), 0 * d)
    if name == "quadratic":
        w = torch.where(t < 0.5, 0.75 - t * t, 0.5 * (1.5 - t).clamp(min=0) ** 2)
        return w, torch.where(t < 0.5, -2 * d, torch.where(t < 1.5, d - 1.5 * torch.sign(d), 0 * d))
    w = torch.where(t < 1, 0.5 * t ** 3 - t * t + 2.0 / 3.0, (2 - t).clamp(min=0) ** 3 / 6)
    return w, torch.where(t < 1, d * (1.5 * t - 2), torch.where(t < 2, -0.5 * torch.sign(d) * (2 - t) ** 2, 0 * d))


def _svd(A):
    """A = U diag(s) V^T of a batch of 3x3 matrices, U and V rotations, by cyclic Jacobi on A^T A."""
    S = A.transpose(1, 2) @ A
    V = torch.eye(3, dtype=A.dtype, device=A.device).expand_as(A).clone()
    for _ in range(8):
        for p, q in ((0, 1), (0, 2), (1, 2)):
            th = 0.5 * torch.atan2(2 * S[:, p, q], S[:, p, p] - S[:, q, q])
            c, s = torch.cos(th)[:, None], torch.sin(th)[:, None]
            for M in (S, V):
                a, b = M[:, :, p].clone(), M[:, :, q].clone()
                M[:, :, p], M[:, :, q] = c * a + s * b, c * b - s * a
            a, b = S[:, p, :].clone(), S[:, q, :].clone()
            S[:, p, :], S[:, q, :] = c * a + s * b, c * b - s * a
    B = A @ V
    s = B.norm(dim=1)
    U = B / s[:, None, :]
    U[:, :, 2] = torch.linalg.cross(U[:, :, 0], U[:, :, 1])
    s = torch.stack([s[:, 0], s[:, 1], (U[:, :, 2] * B[:, :, 2]).sum(1)], 1)
    return U, s, V


def _diag(U, s, V):
    return (U * s[:, None, :]) @ V.transpose(1, 2)


def _friction(vel, normal, hit, friction, surface=0.0):
    """The friction law of a boundary with (not necessarily unit) normals at the rows where `hit`."""
    rel = vel - surface
    vn = (rel * normal).sum(1, keepdim=True)
    vt = rel - vn * normal
    vtn = vt.norm(dim=1, keepdim=True)
    slide = vt + friction * vn * vt / vtn.clamp(min=1e-300)
    out = torch.where(vtn <= -friction * vn + FLT_EPS, torch.zeros_like(rel), slide) + surface
    return torch.where(hit[:, None] & (vn < FLT_EPS), out, vel)


class _Solve64:
    """The snow step on plain 64-bit tensors: explicit or semi-implicit, PIC-FLIP or APIC."""

    def __init__(self, case, sc, obj):
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        t = lambda a: torch.from_numpy(np.array(a)).to(self.dev, torch.float64)  # noqa: E731
        p, d = sc.particles, sc.desc()
        self.case, self.n, self.res = case, p.n, sc.resolution[0]
        self.x, self.v, self.m = t(p.positions), t(p.velocities), t(p.mass)
        self.h, self.dt_max, self.g, self.blend, self.fr = d.stride, d.dt, d.gravity, d.blend, d.friction
        self.apic = d.transfer == _abi.TRANSFER_APIC
        self.S = NODES[case["spline"]]
        self.dinv = {2: 0.0, 3: 4.0, 4: 3.0}[self.S] / self.h ** 2
        f32 = lambda x: float(np.float32(x))  # noqa: E731
        cols = [[f32(m.youngs_modulus / (2 * (1 + m.poisson_ratio))) for m in p.materials],
                [f32(m.youngs_modulus * m.poisson_ratio / ((1 + m.poisson_ratio) * (1 - 2 * m.poisson_ratio)))
                 for m in p.materials], [f32(m.hardening) for m in p.materials],
                [f32(m.critical_compression) for m in p.materials], [f32(m.critical_stretch) for m in p.materials]]
        ids = torch.from_numpy(np.zeros(p.n, np.int64) if p.material is None else p.material.astype(np.int64))
        self.mu0, self.la0, self.xi, self.tc, self.ts = (t(c)[ids.to(self.dev)] for c in cols)
        eye = torch.eye(3, dtype=torch.float64, device=self.dev)
        self.eye = eye
        self.Fe, self.Fp = eye.repeat(p.n, 1, 1), eye.repeat(p.n, 1, 1)
        self.B = torch.zeros_like(self.Fe)
        self.phi = None if obj is None else (t(obj.level_set), f32(obj.friction))
        r = self.res
        z, y, x = torch.meshgrid(*(torch.arange(r, device=self.dev),) * 3, indexing="ij")
        self.idx = torch.stack([x, y, z], -1).reshape(-1, 3).double()
        self.nodes = r ** 3
        self.V0 = torch.zeros_like(self.m)
        self.stencil()
        dens = self.gather(lambda w, g, d: w[:, None], self.density()[:, None])[:, 0]
        self.V0 = self.m / dens

    def stencil(self):
        h, S = self.h, self.S
        base = torch.ceil(self.x / h - {2: 1.0, 3: 1.5, 4: 2.0}[S])
        self.base = base.long()
        ws = [_spline(self.case["spline"], self.x / h - base - k) for k in range(S)]
        self.w, self.dw = torch.stack([w for w, _ in ws], 2), torch.stack([w for _, w in ws], 2)

    def each(self):
        """(node index, weight, gradient, x_node - x_p) of every stencil offset; nodes off the grid get no weight."""
        r, w, dw = self.res, self.w, self.dw
        for c in range(self.S):
            for b in range(self.S):
                for a in range(self.S):
                    i = self.base + torch.tensor([a, b, c], device=self.dev)
                    on = ((i >= 0) & (i < r)).all(1)
                    node = torch.where(on, i[:, 0] + r * (i[:, 1] + r * i[:, 2]), 0)
                    wa, wb, wc = w[:, 0, a], w[:, 1, b], w[:, 2, c]
                    g = torch.stack([dw[:, 0, a] * wb * wc, wa * dw[:, 1, b] * wc, wa * wb * dw[:, 2, c]], 1) / self.h
                    yield node, wa * wb * wc * on, g * on[:, None], i.double() * self.h - self.x

    def scatter(self, f, comps):
        out = torch.zeros((self.nodes, comps), dtype=torch.float64, device=self.dev)
        for node, w, g, d in self.each():
            out.index_add_(0, node, f(w, g, d))
        return out

    def gather(self, f, grid):
        out = 0.0
        for node, w, g, d in self.each():
            k = f(w, g, d)
            v = grid[node]
            out = out + (k * v if k.shape[1] == 1 else (v[:, :, None] * k[:, None, :]).flatten(1))
        return out

    def density(self):
        return self.scatter(lambda w, g, d: (self.m * w)[:, None], 1)[:, 0] / self.h ** 3

    def lame(self):
        f = torch.exp(self.xi * (1 - torch.linalg.det(self.Fp)))
        return (self.mu0 * f)[:, None, None], (self.la0 * f)[:, None, None]

    def stress(self):
        """V0 dPsi/dFe Fe^T."""
        mu, la = self.lame()
        U, s, V = _svd(self.Fe)
        if self.case["neo_hookean"]:
            self.Fe = _diag(U, s.clamp(min=FLT_EPS), V)
            J = torch.linalg.det(self.Fe)[:, None, None]
            t = mu * (self.Fe @ self.Fe.transpose(1, 2) - self.eye) + la * torch.log(J) * self.eye
        else:
            J = torch.linalg.det(self.Fe)[:, None, None]
            t = 2 * mu * (self.Fe - U @ V.transpose(1, 2)) @ self.Fe.transpose(1, 2) + la * (J - 1) * J * self.eye
        return self.V0[:, None, None] * t

    def collide(self, pos, vel):
        lo, hi = FLT_EPS, self.res * self.h - FLT_EPS
        normal = (pos <= lo).double() - (pos >= hi).double()
        return _friction(vel, normal, ((pos <= lo) | (pos >= hi)).any(1), self.fr)

    def collide_object(self, x, vel, dt):
        if self.phi is None:
            return vel
        phi, friction = self.phi
        g = ((x + dt * vel) / self.h).clamp(0, self.res - 1)
        i = g.long().clamp(max=self.res - 2)
        f = g - i
        val, grad = 0.0, 0.0
        for k in range(8):
            d = torch.tensor([k & 1, k >> 1 & 1, k >> 2 & 1], device=self.dev)
            j = i + d
            c = phi.reshape(-1)[j[:, 0] + self.res * (j[:, 1] + self.res * j[:, 2])]
            w, s = torch.where(d.bool(), f, 1 - f), 2.0 * d - 1
            val = val + c * w.prod(1)
            grad = grad + c[:, None] * torch.stack([s[0] * w[:, 1] * w[:, 2], w[:, 0] * s[1] * w[:, 2],
                                                    w[:, 0] * w[:, 1] * s[2]], 1)
        gn = grad.norm(dim=1, keepdim=True)
        return _friction(vel, grad / gn.clamp(min=1e-300), (val <= 0) & (gn[:, 0] > 0), friction)

    def boundary(self, vs, dt):
        if self.case["sticky"]:
            wall = ((self.idx < 3) | (self.idx >= self.res - 3)).any(1)
            vs = torch.where(wall[:, None], torch.zeros_like(vs), vs)
        else:
            vs = self.collide(self.idx * self.h + dt * vs, vs)
        return self.collide_object(self.idx * self.h, vs, dt)

    def hessian(self, u, svd):
        """The elastic energy's Hessian applied to node vectors."""
        G = self.gather(lambda w, g, d: g, u).view(-1, 3, 3)
        F, dF = self.Fe, G @ self.Fe
        mu, la = self.lame()
        J = torch.linalg.det(F)[:, None, None]
        Fi = torch.linalg.inv(F)
        C = J * Fi.transpose(1, 2)
        if self.case["neo_hookean"]:
            FiT = Fi.transpose(1, 2)
            dln = (FiT * dF).sum((1, 2))[:, None, None]
            dP = mu * dF - (la * torch.log(J) - mu) * (FiT @ dF.transpose(1, 2) @ FiT) + la * dln * FiT
        else:
            U, s, V = svd
            M = U.transpose(1, 2) @ dF @ V
            W = (M - M.transpose(1, 2)) / (s[:, :, None] + s[:, None, :])
            dJ = (C * dF).sum((1, 2))[:, None, None]
            tr = (Fi @ dF).diagonal(dim1=1, dim2=2).sum(1)[:, None, None]
            dC = C * tr - C @ dF.transpose(1, 2) @ Fi.transpose(1, 2)
            dP = 2 * mu * (dF - U @ W @ V.transpose(1, 2)) + la * (dJ * C + (J - 1) * dC)
        T = self.V0[:, None, None] * dP @ F.transpose(1, 2)
        return self.scatter(lambda w, g, d: (T @ g[:, :, None])[:, :, 0], 3)

    def solve(self, vs, m, dt):
        """(M + beta dt^2 H) v = M v* by conjugate residual, z = M^-1 r."""
        svd, c, on = _svd(self.Fe), self.case["beta"] * dt * dt, (m > FLT_EPS)[:, None]
        M = torch.where(on[:, 0], m, torch.ones_like(m))[:, None]
        A = lambda u: torch.where(on, M * u + c * self.hessian(u, svd), 0 * u)  # noqa: E731
        x = torch.where(on, vs, 0 * vs)
        b = M * x
        r = b - A(x)
        z = r / M
        p, Az = z.clone(), A(z)
        Ap, zAz = Az.clone(), (z * Az).sum()
        for _ in range(200):
            if r.norm() <= 1e-11 * b.norm():
                break
            al = zAz / (Ap * Ap / M).sum()
            x, r, z = x + al * p, r - al * Ap, z - al * Ap / M
            Az = A(z)
            new = (z * Az).sum()
            p, Ap, zAz = z + new / zAz * p, Az + new / zAz * Ap, new
        return torch.where(on, x, vs)

    def step(self):
        case, dt = self.case, self.dt_max
        if "cfl" in case:
            dt = min(dt, float(np.float32(case["cfl"])) * self.h / float(self.v.norm(dim=1).max()))
        self.stencil()
        tau, C = self.stress(), self.B * self.dinv
        mom = lambda d: self.v + (C @ d[:, :, None])[:, :, 0] if self.apic else self.v  # noqa: E731
        grid = self.scatter(lambda w, g, d: torch.cat([(self.m * w)[:, None], (self.m * w)[:, None] * mom(d),
                                                       -(tau @ g[:, :, None])[:, :, 0]], 1), 7)
        m, on = grid[:, 0], grid[:, :1] > FLT_EPS
        safe = torch.where(on, grid[:, :1], torch.ones_like(grid[:, :1]))
        f = grid[:, 4:] - m[:, None] * torch.tensor([0.0, self.g, 0.0], dtype=torch.float64, device=self.dev)
        vo = torch.where(on, grid[:, 1:4] / safe, grid[:, 1:4])
        vs = torch.where(on, vo + dt * f / safe, torch.zeros_like(vo))
        vs = self.boundary(vs, dt)
        if case["form"] == "implicit":
            vs = self.boundary(self.solve(vs, m, dt), dt)
        pic = self.gather(lambda w, g, d: w[:, None], vs)
        gv = self.gather(lambda w, g, d: g, vs).view(-1, 3, 3)
        if self.apic:
            self.B = self.gather(lambda w, g, d: w[:, None] * d, vs).view(-1, 3, 3)
            self.v = pic
        else:
            flip = self.v + self.gather(lambda w, g, d: w[:, None], vs - vo)
            self.v = self.blend * flip + (1 - self.blend) * pic
        Fe = (self.eye + dt * gv) @ self.Fe
        U, s, V = _svd(Fe)
        c = torch.maximum(torch.minimum(s, 1 + self.ts[:, None]), 1 - self.tc[:, None])
        F = Fe @ self.Fp
        self.Fe, self.Fp = _diag(U, c, V), _diag(V, 1 / c, U) @ F
        if case["form"] == "objects":
            self.v = self.collide(self.x + dt * self.v, self.v)
            self.v = self.collide_object(self.x, self.v, dt)
        self.x = self.x + dt * self.v


def exact(case, seed):
    scenes = _scenes(case, seed)
    cost = sum(s.n for s in scenes) * NODES[case["spline"]] ** 3 * case["steps"] * (30 if case["form"] == "implicit"
                                                                                    else 1)
    if cost > 1.2e9:
        return None
    got = {"position": [], "velocity": [], "det_fe": [], "density": []}
    for sc in scenes:
        s = _Solve64(case, sc, _object(sc) if case["form"] == "objects" else None)
        for _ in range(case["steps"]):
            s.step()
        got["position"].append(s.x)
        got["velocity"].append(s.v)
        got["det_fe"].append(torch.linalg.det(s.Fe))
        if case["form"] == "export":
            s.stencil()
            got["density"].append(s.density().view(s.res, s.res, s.res))
    return {k: torch.cat(v).cpu() for k, v in got.items() if v}
