"""The work that users of the framework have it do, as cases that can be timed.

Each case names a `kind` (one public entry point or a user's sequence of them),
a scene, its sizes and the options that are used in earnest.  Scenes follow the
repository's own generators (dam break, pool drop with a static sphere, blob
scene with a box obstacle), made here on the GPU:

  project      solve + velocity update, CUDA tensors (VariationalPressureSolver / NormalPressureSolver .project)
  solve_host   the same solve from a simulator's own pageable FP64 host arrays (.solve)
  batch        many uneven scenes per call (BatchProjector.project)
  backward     the projection's adjoint (.backward)
  rollout      advect + project steps and their gradient (Rollout.forward / .backward)
  extrapolate  velocity extrapolation after the projection (.extrapolateVelocity)
  p2g          particles to faces (ParticleSteps.updateVelocityByParticles)
  field        distance field and its classification (ParticleSteps.updateField)
  step         one whole simulator time step (Simulation.time_step)
"""
import math

import numpy as np
import torch

AIR, FLUID, SOLID = 0, 1, 2
DEV = "cuda"


def listed():
    return [
        # the smallest call: a preview-size projection, where launches and waits count
        {"name": "project_small", "kind": "project", "scene": "blob", "ni": 24, "nj": 20, "nk": 22, "matrix": "variational",
         "precision": "f64", "io": "f64", "fractional": False, "tol": 1e-6, "max_iter": 200},
        # the drop-in inside a CPU simulator: its own 64^3 dam break from pageable host arrays, FP64
        {"name": "solve_host_dam64", "kind": "solve_host", "scene": "dam", "ni": 64, "nj": 64, "nk": 64, "tol": 1e-6, "max_iter": 200},
        # the reference's arithmetic on a mid-size device-resident grid
        {"name": "project_dam128_f64", "kind": "project", "scene": "dam", "ni": 128, "nj": 128, "nk": 128, "matrix": "variational",
         "precision": "f64", "io": "f64", "fractional": False, "tol": 1e-6, "max_iter": 300},
        # a ragged pool with a static sphere's fractional faces
        {"name": "project_pool_ragged", "kind": "project", "scene": "pool", "ni": 150, "nj": 97, "nk": 131, "matrix": "variational",
         "precision": "mixed", "io": "f32", "fractional": True, "tol": 1e-6, "max_iter": 300},
        # the headline projection: 256^3 blobs, mixed precision
        {"name": "project_blob256", "kind": "project", "scene": "blob", "ni": 256, "nj": 256, "nk": 256, "matrix": "variational",
         "precision": "mixed", "io": "f32", "fractional": False, "tol": 1e-6, "max_iter": 200},
        # many independent uneven scenes in one call
        {"name": "batch_uneven12", "kind": "batch", "count": 12, "lo": 32, "hi": 160, "precision": "mixed", "tol": 1e-6, "max_iter": 200},
        # the adjoint of one projection, as a training step calls it
        {"name": "backward_blob128", "kind": "backward", "scene": "blob", "ni": 128, "nj": 128, "nk": 128, "precision": "mixed",
         "io": "f32", "fractional": True, "tol": 1e-6, "max_iter": 200},
        # a differentiable rollout with its gradient, FP64
        {"name": "rollout_dam48", "kind": "rollout", "ni": 48, "nj": 48, "nk": 48, "steps": 2, "every": 2},
        # the velocity extrapolation of a large grid (CFL 1: 6 layers)
        {"name": "extrapolate_192", "kind": "extrapolate", "scene": "blob", "ni": 192, "nj": 192, "nk": 192, "io": "f32", "layers": 6},
        # particles to faces, eight particles per fluid cell
        {"name": "p2g_dam96", "kind": "p2g", "scene": "dam", "ni": 96, "nj": 96, "nk": 96},
        # the distance field at the simulator's two vertices per cell
        {"name": "field_dam96", "kind": "field", "scene": "dam", "ni": 96, "nj": 96, "nk": 96, "subdiv": 2},
        # one whole simulator time step: 128^3 pool drop, CFL 5 (10 extrapolation layers), FP64
        {"name": "step_pool128", "kind": "step", "scene": "pool", "ni": 128, "nj": 128, "nk": 128, "cfl": 5.0, "tol": 1e-6, "max_iter": 200},
    ]


def _dims(rng, lo, hi):
    """Three sizes, log-uniform in [lo, hi]: a common scale and an aspect per axis, so odd and uneven ones appear."""
    s = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return {k: int(min(hi, max(lo, round(s * math.exp(rng.uniform(-0.3, 0.3)))))) for k in ("ni", "nj", "nk")}


def draw(rng):
    kind = rng.choice(["project", "project", "project", "solve_host", "batch", "backward", "rollout", "extrapolate", "p2g", "field", "step"])
    c = {"kind": kind}
    if kind == "project":
        c["scene"] = rng.choice(["dam", "pool", "blob"])
        c["precision"] = rng.choice(["f64", "mixed", "mixed", "f32"])
        c |= _dims(rng, 20, 144 if c["precision"] == "f64" else 224)
        c["io"] = "f64" if c["precision"] == "f64" else "f32"
        c["matrix"] = rng.choice(["variational", "variational", "variational", "normal"])
        c["fractional"] = c["matrix"] == "variational" and c["scene"] != "dam" and rng.random() < 0.5
        c |= {"tol": 1e-6, "max_iter": 400}
    elif kind == "solve_host":
        c |= {"scene": rng.choice(["dam", "pool"]), **_dims(rng, 24, 96), "tol": 1e-6, "max_iter": 300}
    elif kind == "batch":
        lo = rng.choice([24, 32, 48])
        c |= {"count": rng.randint(4, 14), "lo": lo, "hi": rng.randint(lo + 16, 144), "precision": rng.choice(["mixed", "f64"]),
              "tol": 1e-6, "max_iter": 300}
    elif kind == "backward":
        c |= {"scene": rng.choice(["pool", "blob"]), **_dims(rng, 24, 144), "precision": rng.choice(["mixed", "f64"]), "tol": 1e-6,
              "max_iter": 300, "fractional": rng.random() < 0.5}
        c["io"] = "f64" if c["precision"] == "f64" else "f32"
    elif kind == "rollout":
        c |= {**_dims(rng, 24, 56), "steps": rng.choice([2, 3]), "every": rng.choice([1, 2])}
    elif kind == "extrapolate":
        c |= {"scene": rng.choice(["dam", "pool", "blob"]), **_dims(rng, 24, 224), "io": rng.choice(["f32", "f64"]), "layers": rng.randint(3, 10)}
    elif kind in ("p2g", "field"):
        c |= {"scene": rng.choice(["dam", "pool"]), **_dims(rng, 24, 112)}
        if kind == "field":
            c["subdiv"] = rng.choice([2, 2, 3])
    else:
        c |= {"scene": rng.choice(["dam", "pool"]), **_dims(rng, 32, 112), "cfl": rng.choice([1.0, 5.0]), "tol": 1e-6, "max_iter": 300}
    return c


# ---------------------------------------------------------------- scenes
def _centres(n):
    return (torch.arange(n, device=DEV, dtype=torch.float64) + 0.5) / n


def _xyz(dims):
    ni, nj, nk = dims
    return _centres(ni)[None, None, :], _centres(nj)[None, :, None], _centres(nk)[:, None, None]


def _border(mat):
    mat[0], mat[-1] = SOLID, SOLID
    mat[:, 0], mat[:, -1] = SOLID, SOLID
    mat[:, :, 0], mat[:, :, -1] = SOLID, SOLID


def _box_weights(dims, lo, hi):
    """Open fraction of every face against a solid box (x, y, z extents lo..hi)."""
    over = []
    inside = []
    for n, a, b in zip(dims, lo, hi):
        e = torch.arange(n + 1, device=DEV, dtype=torch.float64) / n
        over.append((torch.minimum(e[1:], torch.tensor(b, device=DEV)) - torch.maximum(e[:-1], torch.tensor(a, device=DEV))).clamp_min(0.0) * n)
        inside.append(((e > a) & (e < b)).double())
    (ox, oy, oz), (ix, iy, iz) = over, inside
    tri = lambda x, y, z: 1.0 - z[:, None, None] * y[None, :, None] * x[None, None, :]  # noqa: E731
    return tri(ix, oy, oz), tri(ox, iy, oz), tri(ox, oy, iz)


def _sphere_weights(dims, centre, radius, sub=4):
    """Open fraction of every face against a solid sphere, by sub x sub points on the face."""
    out = []
    off = [(q + 0.5) / sub for q in range(sub)]
    for axis in range(3):
        acc = None
        for a in off:
            for b in off:
                shift = {0: (0.0, a, b), 1: (a, 0.0, b), 2: (a, b, 0.0)}[axis]
                d2 = [((torch.arange(n + (q == axis), device=DEV, dtype=torch.float64) + shift[q]) / n - centre[q]) ** 2
                      for q, n in enumerate(dims)]
                hit = (d2[0][None, None, :] + d2[1][None, :, None] + d2[2][:, None, None] < radius * radius).double()
                acc = hit if acc is None else acc + hit
        out.append(1.0 - acc / (sub * sub))
    return tuple(out)


def _scene(kind, dims, seed, dtype, fractional=False, noise=0.5):
    """mat and faces (u, v, w), and face weights where asked for; all from the seed."""
    ni, nj, nk = dims
    host = np.random.default_rng(seed)
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    x, y, z = _xyz(dims)
    mat = torch.zeros((nk, nj, ni), dtype=torch.uint8, device=DEV)
    weights = None
    if kind == "blob":
        phi = torch.zeros((nk, nj, ni), dtype=torch.float64, device=DEV)
        cen, sig = host.uniform(0.0, 1.0, (32, 3)), host.uniform(0.03, 0.12, 32)
        for c, s in zip(cen, sig):
            g = [torch.exp(-(t - float(q)) ** 2 / (2.0 * float(s) * float(s))) for t, q in zip((x, y, z), c)]
            phi += g[2] * (g[1] * g[0])
        mat[phi > 0.5] = FLUID
        sx, sy = host.uniform(0.35, 0.65, 2)
        side = np.array([sx, sy, min(0.95, 0.10 / (sx * sy))])
        lo = host.uniform(0.0, 1.0 - side)
        hi = lo + side
        mat[(x > lo[0]) & (x < hi[0]) & (y > lo[1]) & (y < hi[1]) & (z > lo[2]) & (z < hi[2])] = SOLID
        if fractional:
            weights = _box_weights(dims, lo, hi)
        noise = 1.0
    else:
        # the free surface starts at a level of the seed's own, a few cells around the usual one
        level = float(host.uniform(-0.03, 0.03))
        if kind == "dam":
            mat[((x < 0.4 + level) & (y < 0.5 - level)).expand(nk, nj, ni)] = FLUID
        else:
            mat[(y < 0.3 + level) | ((x - 0.5) ** 2 + (y - 0.7) ** 2 + (z - 0.5) ** 2 < 0.15 ** 2)] = FLUID
            mat[(x - 0.3) ** 2 + (y - 0.2) ** 2 + (z - 0.5) ** 2 < 0.1 ** 2] = SOLID
            if fractional:
                weights = _sphere_weights(dims, (0.3, 0.2, 0.5), 0.1)
    _border(mat)
    shapes = ((nk, nj, ni + 1), (nk, nj + 1, ni), (nk + 1, nj, ni))
    faces = [(torch.rand(s, generator=gen, device=DEV, dtype=torch.float64) * 2.0 - 1.0) * noise for s in shapes]
    if kind != "blob":
        # gravity's impulse on the faces that border fluid
        fl = mat == FLUID
        wet = torch.zeros(shapes[1], dtype=torch.bool, device=DEV)
        wet[:, :-1] |= fl
        wet[:, 1:] |= fl
        faces[1][wet] -= 9.8 / 30.0
    faces = tuple(f.to(dtype).contiguous() for f in faces)
    if weights is not None:
        weights = tuple(w.to(dtype).contiguous() for w in weights)
    return mat, faces, weights


def _particles(mat, dx, seed):
    """Eight particles per fluid cell at the centre +- dx/4, jittered, with U[-1, 1] velocities: (n, 6) rows of position and velocity."""
    gen = torch.Generator(device=DEV).manual_seed(int(seed) + 1)
    kji = torch.nonzero(mat == FLUID).double()
    c = (kji.flip(1) + 0.5) * dx
    off = torch.tensor([(a, b, d) for a in (-1, 1) for b in (-1, 1) for d in (-1, 1)], device=DEV, dtype=torch.float64) * (0.25 * dx)
    p = (c[:, None, :] + off[None]).reshape(-1, 3)
    p = p + (torch.rand(p.shape, generator=gen, device=DEV, dtype=torch.float64) * 2 - 1) * (0.2 * dx)
    v = torch.rand(p.shape, generator=gen, device=DEV, dtype=torch.float64) * 2 - 1
    return torch.cat([p, v], 1).contiguous()


def _case_dims(c):
    return c["ni"], c["nj"], c["nk"]


def _type(c):
    return torch.float64 if c.get("io", "f64") == "f64" else torch.float32


def _batch_scenes(c, seed):
    r = np.random.default_rng([c["count"], c["lo"], c["hi"]])   # a batch keeps its sizes; its scenes are the seed's
    kind = torch.float64 if c["precision"] == "f64" else torch.float32
    return [_scene("blob", tuple(int(v) for v in r.integers(c["lo"], c["hi"] + 1, 3)), seed * 1000 + q, kind) for q in range(c["count"])]


def _gradient_faces(c, seed):
    gen = torch.Generator(device=DEV).manual_seed(int(seed) + 2)
    ni, nj, nk = _case_dims(c)
    return tuple((torch.rand(s, generator=gen, device=DEV, dtype=torch.float64) * 2 - 1).to(_type(c))
                 for s in ((nk, nj, ni + 1), (nk, nj + 1, ni), (nk + 1, nj, ni)))


_BOX = ((0.1037, 0.3461), (0.1037, 0.4483), (0.2019, 0.7989))   # the rollout's loss box, inside the dam; its sides meet no face position


def _radius(dx):
    """FluidSimulator's field radius: three times its particle radius."""
    return 3.0 * (3 * (dx ** 3 / 8.0) / (4 * 3.141592653)) ** (1.0 / 3.0)


# ---------------------------------------------------------------- prepare / run
def prepare(case, seed):
    from xfluid_b200.batch import BatchProjector
    from xfluid_b200.particles import ParticleSteps
    from xfluid_b200.rollout import Rollout
    from xfluid_b200.simulation import Simulation
    from xfluid_b200.solver import NormalPressureSolver, VariationalPressureSolver

    c, kind = case, case["kind"]
    s = {"kind": kind, "case": c}
    if kind == "batch":
        scenes = _batch_scenes(c, seed)
        s["solver"] = BatchProjector(precision=c["precision"], tol=c["tol"], max_iter=c["max_iter"])
        s["faces0"] = [f for _, f, _ in scenes]
        s["scenes"] = [{"mat": m, "u": f[0].clone(), "v": f[1].clone(), "w": f[2].clone(), "pressure": torch.zeros(m.shape, dtype=f[0].dtype, device=DEV)}
                       for m, f, _ in scenes]
        return s
    if kind == "rollout":
        mat, faces, _ = _scene("dam", _case_dims(c), seed, torch.float64)
        s["faces0"] = faces
        s["rollout"] = Rollout(mat, steps=c["steps"], checkpoint_every=c["every"], dt_over_dx=0.5, box=_BOX)
        return s
    if kind in ("p2g", "field"):
        ni, nj, nk = _case_dims(c)
        dx = 1.0 / ni
        mat, faces, _ = _scene(c["scene"], (ni, nj, nk), seed, torch.float64)
        s["steps"], s["mat"], s["parts"] = ParticleSteps(dx), mat, _particles(mat, dx, seed)
        s["faces"] = faces
        if kind == "field":
            s["mat0"] = mat.clone()
            s["phi"] = torch.zeros((nk * c["subdiv"] + 1, nj * c["subdiv"] + 1, ni * c["subdiv"] + 1), dtype=torch.float64, device=DEV)
        return s
    if kind == "step":
        ni, nj, nk = _case_dims(c)
        dx = 1.0 / ni
        mat, faces, _ = _scene(c["scene"], (ni, nj, nk), seed, torch.float64)
        parts = _particles(mat, dx, seed)
        sim = Simulation(mat.clone(), parts.clone(), dx, cfl=c["cfl"], tol=c["tol"], max_iter=c["max_iter"])
        sim.steps.updateVelocityByParticles(sim.particles, (sim.u, sim.v, sim.w))
        s["sim"], s["mat0"], s["parts0"] = sim, mat, parts
        s["faces0"] = (sim.u.clone(), sim.v.clone(), sim.w.clone())
        s["dt"] = min(1.0 / 30.0, c["cfl"] * dx / math.sqrt(3.0))
        return s
    dims = _case_dims(c)
    dtype = torch.float64 if kind == "solve_host" else _type(c)
    mat, faces, weights = _scene(c["scene"], dims, seed, dtype, c.get("fractional", False))
    cls = NormalPressureSolver if c.get("matrix") == "normal" else VariationalPressureSolver
    solver = cls(c.get("precision", "f64"), tol=c.get("tol", 1e-6), max_iter=c.get("max_iter", 200))
    solver.setSize(*dims)
    s["solver"] = solver
    if kind == "solve_host":
        mat, faces = mat.cpu().numpy(), tuple(f.cpu().numpy() for f in faces)
        s["p"] = np.zeros(mat.shape)
    else:
        s["faces0"] = faces
        faces = tuple(f.clone() for f in faces)
        s["p"] = torch.zeros(mat.shape, dtype=dtype, device=DEV)
    s["mat"], s["faces"] = mat, faces
    solver.setMaterial(mat)
    solver.setVelocityField(*faces)
    if weights is not None:
        solver.setFaceWeights(*weights)
    if kind == "backward":
        s["g"] = _gradient_faces(c, seed)
        s["d"] = tuple(torch.empty_like(g) for g in s["g"])
    return s


def run(state):
    s, kind = state, state["kind"]
    if kind == "project":
        for f, f0 in zip(s["faces"], s["faces0"]):   # a step's new velocities arrive
            f.copy_(f0)
        s["solver"].project(s["p"])
        return {"p": s["p"], "u": s["faces"][0], "v": s["faces"][1], "w": s["faces"][2]}
    if kind == "solve_host":
        s["solver"].solve(s["p"])
        return s["p"]
    if kind == "batch":
        for sc, f0 in zip(s["scenes"], s["faces0"]):
            for k, f in zip("uvw", f0):
                sc[k].copy_(f)
        s["solver"].project(s["scenes"])
        return [[sc["pressure"], sc["u"], sc["v"], sc["w"]] for sc in s["scenes"]]
    if kind == "backward":
        s["solver"].backward(*s["g"], *s["d"])
        return list(s["d"])
    if kind == "rollout":
        loss = s["rollout"].forward(*s["faces0"])
        return [loss, *s["rollout"].backward()]
    if kind == "extrapolate":
        for f, f0 in zip(s["faces"], s["faces0"]):
            f.copy_(f0)
        s["solver"].extrapolateVelocity(s["case"]["layers"])
        return list(s["faces"])
    if kind == "p2g":
        s["steps"].updateVelocityByParticles(s["parts"], s["faces"])
        return list(s["faces"])
    if kind == "field":
        s["mat"].copy_(s["mat0"])
        s["steps"].updateField(s["parts"], s["mat"], subdiv=s["case"]["subdiv"], phi=s["phi"])
        return [s["phi"], s["mat"]]
    sim = s["sim"]
    sim.set_state(particles=s["parts0"], uvw=s["faces0"], mat=s["mat0"])
    sim.time_step(s["dt"])
    return {"particles": sim.particles, "u": sim.u, "v": sim.v, "w": sim.w, "p": sim.pressure, "phi": sim.phi, "mat": sim.mat}


# ---------------------------------------------------------------- work
def work(case):
    """Inputs read once and outputs written once; the operations of the passes a solver cannot do without are not counted."""
    c, kind = case, case["kind"]
    if kind == "batch":
        n = ((c["lo"] + c["hi"]) / 2.0) ** 3 * c["count"]
        b = 8 if c["precision"] == "f64" else 4
        return {"bytes": n * (1 + 6 * b + b), "flops": n * 20}
    ni, nj, nk = _case_dims(c)
    n = float(ni * nj * nk)
    share = {"dam": 0.2, "pool": 0.3, "blob": 0.15}[c.get("scene", "dam")]
    parts = 8 * share * n
    b = 8 if kind == "solve_host" or c.get("io", "f64") == "f64" else 4
    faces = 3 * n * b
    if kind == "project":
        return {"bytes": n + 2 * faces + n * b + (faces if c["fractional"] else 0), "flops": 20 * n * share}
    if kind == "solve_host":
        return {"bytes": n + faces + n * b, "flops": 20 * n * share}
    if kind == "backward":
        return {"bytes": n + 2 * faces + (faces if c["fractional"] else 0), "flops": 20 * n * share}
    if kind == "rollout":
        return {"bytes": (n + 4 * faces) * 2 * c["steps"], "flops": 200 * n * c["steps"]}
    if kind == "extrapolate":
        return {"bytes": n + 2 * faces, "flops": 6 * n}
    if kind == "p2g":
        return {"bytes": 48 * parts + faces, "flops": 3 * 27 * 16 * parts}
    if kind == "field":
        v = n * c["subdiv"] ** 3
        return {"bytes": 24 * parts + 8 * v + 2 * n, "flops": 14 * parts * 4.2 * (0.93 * c["subdiv"]) ** 3}
    return {"bytes": 2 * 48 * parts + 2 * n + 2 * faces + 8 * n + 64 * n, "flops": 3 * 27 * 16 * parts + 500 * parts}


# ---------------------------------------------------------------- the same in 64 bits
def _faces_of(mat, axis):
    """Left and right cell's material of the faces that lie between two cells on `axis` (0 x, 1 y, 2 z), and the slices of the two cells."""
    d = 2 - axis
    n = mat.shape[d]
    return mat.narrow(d, 0, n - 1), mat.narrow(d, 1, n - 1), d


class _System:
    """The pressure system on the dense grid: per inner face the coefficient, the right-hand side's factor and the gradient's factor."""

    def __init__(self, mat, weights, matrix):
        self.mat, self.normal = mat, matrix == "normal"
        fl = mat == FLUID
        near = torch.zeros_like(fl)
        self.cf, self.bf, self.gf, self.mirror = [], [], [], []
        for axis in range(3):
            l, r, d = _faces_of(mat, axis)
            n = mat.shape[d]
            ff, fs, fa = (l == FLUID) & (r == FLUID), None, None
            fs = ((l == FLUID) & (r == SOLID)) | ((l == SOLID) & (r == FLUID))
            fa = ((l == FLUID) & (r == AIR)) | ((l == AIR) & (r == FLUID))
            m = weights[axis].narrow(d, 1, n - 1).double() if weights is not None else torch.ones_like(l, dtype=torch.float64)
            if self.normal:
                self.cf.append((ff | fa).double())
                self.bf.append((ff | fa).double())
                self.gf.append((ff | fa).double())
                self.mirror.append(fs)
            else:
                self.cf.append(m * (ff.double() + 0.5 * fs.double() + 2.0 * fa.double()))
                self.bf.append(m * (ff.double() + 0.5 * fs.double() + fa.double()))
                self.gf.append((m != 0).double() * (ff.double() + fs.double() + 2.0 * fa.double()))
                self.mirror.append(None)
            near.narrow(d, 0, n - 1).logical_or_(r == FLUID)
            near.narrow(d, 1, n - 1).logical_or_(l == FLUID)
        self.mask = (fl if self.normal else fl | ((mat == SOLID) & near)).double()
        self.diag = torch.zeros_like(self.mask)
        for axis in range(3):
            d, n = 2 - axis, mat.shape[2 - axis]
            self.diag.narrow(d, 0, n - 1).add_(self.cf[axis])
            self.diag.narrow(d, 1, n - 1).add_(self.cf[axis])
        self.diag *= self.mask

    def apply(self, p):
        y = torch.zeros_like(p)
        for axis in range(3):
            d, n = 2 - axis, p.shape[2 - axis]
            t = self.cf[axis] * (p.narrow(d, 1, n - 1) - p.narrow(d, 0, n - 1))
            y.narrow(d, 0, n - 1).sub_(t)
            y.narrow(d, 1, n - 1).add_(t)
        return y.mul_(self.mask)

    def rhs(self, uvw):
        b = 0.0
        for axis, f in enumerate(uvw):
            d, n = 2 - axis, self.mat.shape[2 - axis]
            t = self.bf[axis] * f.narrow(d, 1, n - 1)
            pad = [0, 0, 0, 0, 0, 0]
            lo, hi = list(pad), list(pad)
            lo[2 * axis], hi[2 * axis + 1] = 1, 1
            b = b + torch.nn.functional.pad(t, lo) - torch.nn.functional.pad(t, hi)
        return b * self.mask

    def solve(self, b, tol=1e-13, most=20000):
        x, r = torch.zeros_like(b), b.clone()
        inv = torch.where(self.diag > 0, 1.0 / self.diag.clamp_min(1e-300), torch.zeros_like(b))
        z = inv * r
        s, rho = z.clone(), (z * r).sum()
        goal = float(b.abs().max()) * tol
        if goal == 0.0:
            return x
        for it in range(most):
            q = self.apply(s)
            a = rho / (q * s).sum()
            x.addcmul_(s, a)
            r.addcmul_(q, -a)
            if it % 25 == 24 and float(r.abs().max()) <= goal:
                break
            z = inv * r
            rho, old = (z * r).sum(), rho
            s.mul_(rho / old).add_(z)
        return x

    def update(self, uvw, p):
        out = []
        for axis, f in enumerate(uvw):
            d, n = 2 - axis, self.mat.shape[2 - axis]
            t = self.gf[axis] * (p.narrow(d, 1, n - 1) - p.narrow(d, 0, n - 1))
            if self.normal:
                t = torch.where(self.mirror[axis], f.narrow(d, 1, n - 1), t)
            pad = [0, 0, 0, 0, 0, 0]
            pad[2 * axis], pad[2 * axis + 1] = 1, 1
            out.append(f - torch.nn.functional.pad(t, pad))
        return out


class _Solve(torch.autograd.Function):
    @staticmethod
    def forward(ctx, b, system):
        ctx.system = system
        return system.solve(b)

    @staticmethod
    def backward(ctx, g):
        return ctx.system.solve(g * ctx.system.mask), None


def _lattice(comp, pos, field):
    """Trilinear sample of face component `comp` at positions in cell units, lattice coordinates clamped to the grid."""
    n = [field.shape[2], field.shape[1], field.shape[0]]
    off = [0.0 if q == comp else 0.5 for q in range(3)]
    at, frac = [], []
    for q in range(3):
        f = (pos[q] - off[q]).clamp(0.0, n[q] - 1.0)
        a = f.detach().floor().clamp(0, max(n[q] - 2, 0))
        at.append(a.long())
        frac.append(f - a)
    flat, total = field.reshape(-1), 0.0
    for q in range(8):
        o = (q & 1, (q >> 1) & 1, q >> 2)
        w = 1.0
        for e in range(3):
            w = w * (frac[e] if o[e] else 1.0 - frac[e])
        total = total + w * flat[((at[2] + o[2]) * n[1] + at[1] + o[1]) * n[0] + at[0] + o[0]]
    return total


def _advect(uvw, c):
    out = []
    for comp, f in enumerate(uvw):
        nk, nj, ni = f.shape
        off = [0.0 if q == comp else 0.5 for q in range(3)]
        ax = [torch.arange(n, device=DEV, dtype=torch.float64) + off[q] for q, n in enumerate((ni, nj, nk))]
        x = [ax[0][None, None, :].expand(f.shape), ax[1][None, :, None].expand(f.shape), ax[2][:, None, None].expand(f.shape)]
        vel = [_lattice(q, x, g) for q, g in enumerate(uvw)]
        out.append(_lattice(comp, [x[q] - c * vel[q] for q in range(3)], f))
    return out


def _wendland(rs, r):
    r2 = r * r
    w = 1.0 - (4.0 / 9.0) * rs ** 3 / r2 ** 3 + (17.0 / 9.0) * rs ** 2 / r2 ** 2 - (22.0 / 9.0) * rs / r2
    return torch.where(rs < r2, w, torch.zeros_like(w))


def _splat(pos, value, ext, unit, r):
    """Sums over the particles of weight and weight * value at the points ((i + 0.5) unit, ...) of a grid of `ext` points."""
    wsum = torch.zeros(ext[0] * ext[1] * ext[2], dtype=torch.float64, device=DEV)
    vsum = torch.zeros_like(wsum) if value is not None else None
    lo = torch.ceil((pos - r) / unit - 0.5).long()
    reach = int(math.floor(2 * r / unit)) + 2
    for a in range(reach):
        for b in range(reach):
            for d in range(reach):
                at = lo + torch.tensor([a, b, d], device=DEV)
                diff = (at.double() + 0.5) * unit - pos
                ok = ((at >= 0) & (at < torch.tensor(ext, device=DEV))).all(1)
                w = torch.where(ok, _wendland((diff * diff).sum(1), r), torch.zeros_like(diff[:, 0]))
                flat = torch.where(ok, (at[:, 2] * ext[1] + at[:, 1]) * ext[0] + at[:, 0], torch.zeros_like(at[:, 0]))
                wsum.index_add_(0, flat, w)
                if value is not None:
                    vsum.index_add_(0, flat, w * value)
    shape = (ext[2], ext[1], ext[0])
    return wsum.view(shape), None if vsum is None else vsum.view(shape)


def _spread(mat, f, axis, layers):
    """Layer by layer outward from the faces of fluid cells, the mean of the neighbours in the layer before."""
    fl = mat == FLUID
    d = 2 - axis
    done = torch.zeros(f.shape, dtype=torch.bool, device=DEV)
    done.narrow(d, 0, mat.shape[d]).logical_or_(fl)
    done.narrow(d, 1, mat.shape[d]).logical_or_(fl)
    f, last = f.clone(), done.clone()
    for _ in range(layers):
        total, count = torch.zeros_like(f), torch.zeros_like(f)
        for e in range(3):
            n = f.shape[e]
            for a, b in ((0, 1), (1, 0)):
                src_f, src = f.narrow(e, b, n - 1), last.narrow(e, b, n - 1)
                total.narrow(e, a, n - 1).add_(torch.where(src, src_f, torch.zeros_like(src_f)))
                count.narrow(e, a, n - 1).add_(src.double())
        last = (count > 0) & ~done
        f = torch.where(last, total / count.clamp_min(1.0), f)
        done = done | last
    return f


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "step":
        return None   # five stages with collisions: its stages are cases of their own
    if kind == "batch":
        out = []
        for mat, faces, _ in _batch_scenes(c, seed):
            system = _System(mat, None, "variational")
            faces = [f.double() for f in faces]
            p = system.solve(system.rhs(faces))
            out.append([p, *system.update(faces, p)])
        return out
    if kind == "rollout":
        mat, faces, _ = _scene("dam", _case_dims(c), seed, torch.float64)
        system = _System(mat, None, "variational")
        start = [f.clone().requires_grad_(True) for f in faces]
        state = start
        for _ in range(c["steps"]):
            state = _advect(state, 0.5)
            state = system.update(state, _Solve.apply(system.rhs(state), system))
        loss = 0.0
        ni, nj, nk = _case_dims(c)
        for comp, f in enumerate(state):
            inside = True
            for q, n in enumerate((ni, nj, nk)):
                x = (torch.arange(n + (q == comp), device=DEV, dtype=torch.float64) + (0.0 if q == comp else 0.5)) / n
                ok = (x >= _BOX[q][0]) & (x <= _BOX[q][1])
                inside = inside & ok.view([1, 1, -1] if q == 0 else [1, -1, 1] if q == 1 else [-1, 1, 1])
            loss = loss + (f * f * inside).sum()
        loss.backward()
        return [float(loss.detach()), *[f.grad for f in start]]
    if kind in ("p2g", "field"):
        ni, nj, nk = _case_dims(c)
        dx = 1.0 / ni
        mat, _, _ = _scene(c["scene"], (ni, nj, nk), seed, torch.float64)
        parts = _particles(mat, dx, seed)
        if kind == "field":
            s = c["subdiv"]
            phi, _ = _splat(parts[:, :3], None, (ni * s + 1, nj * s + 1, nk * s + 1), dx / s, _radius(dx))
            return [phi, None]
        out = []
        for axis in range(3):
            shift = torch.zeros(3, dtype=torch.float64, device=DEV)
            shift[axis] = 0.5 * dx
            ext = tuple(n + (q == axis) for q, n in enumerate((ni, nj, nk)))
            w, v = _splat(parts[:, :3] + shift, parts[:, 3 + axis].contiguous(), ext, dx, 1.5 * dx)
            out.append(torch.where(w > 1e-7, v / w.clamp_min(1e-300), torch.zeros_like(v)))
        return out
    dtype = torch.float64 if kind == "solve_host" else _type(c)
    mat, faces, weights = _scene(c["scene"], _case_dims(c), seed, dtype, c.get("fractional", False))
    faces = [f.double() for f in faces]
    if kind == "extrapolate":
        return [_spread(mat, f, axis, c["layers"]) for axis, f in enumerate(faces)]
    system = _System(mat, weights, c.get("matrix", "variational"))
    if kind == "backward":
        g = [f.double() for f in _gradient_faces(c, seed)]
        probe = [torch.zeros_like(f).requires_grad_(True) for f in g]
        p = _Solve.apply(system.rhs(probe), system)
        sum((a * b).sum() for a, b in zip(system.update(probe, p), g)).backward()
        return [f.grad for f in probe]
    p = system.solve(system.rhs(faces))
    if kind == "solve_host":
        return p.cpu().numpy()
    return dict(zip(("p", "u", "v", "w"), (p, *system.update(faces, p))))
