"""Timed cases of the framework's own entry points.

A case is one call sequence of a user's program: an episode of a scene (``gs.Scene``: reset to a
state, a few steps, read the state back), a batch of scenes advanced together
(``BatchedScenes``), a differentiated rollout (``grad.rollout`` and ``gs.Scene`` with
``requires_grad``), and the signed-distance grid of a tool mesh that a scene build makes.  States
are those of a running simulation: jittered particle lattices in motion with deformation
gradients around the identity, so plastic materials yield and contacts act.

``exact`` steps the same inputs in float64 with plain torch (Stomakhin / Hu MLS-MPM as the
solver documents it: quadratic B-splines, APIC, the materials' return mappings); gradients come
from torch autograd through that restatement.
"""

import math

import numpy as np
import torch

DEV = "cuda"
EPS = float(np.finfo(np.float32).eps)  # gs.EPS at precision "32": part of the model
NU, RHO = 0.2, 1000.0
YOUNG = {"elastic": 3e5, "neohooken": 3e5, "muscle": 3e5, "liquid": 1e5, "sand": 1e6, "snow": 1e6, "elastoplastic": 1e6}
MIXED = ("liquid", "sand", "snow", "elastoplastic")


# ---------------------------------------------------------------- the cases


def _scene(name, material, nx, ny, nz, density, steps, substeps, envs=0, sphere=False):
    c = dict(kind="scene", material=material, nx=nx, ny=ny, nz=nz, density=density, steps=steps, substeps=substeps,
             envs=envs, sphere=sphere)
    return dict(c, name=name) if name else c


def _batch(name, scenes, n_lo, n_hi, substeps):
    c = dict(kind="batch", scenes=scenes, n_lo=n_lo, n_hi=n_hi, substeps=substeps)
    return dict(c, name=name) if name else c


def _grad(name, material, nx, ny, nz, density, substeps, every):
    c = dict(kind="grad", material=material, nx=nx, ny=ny, nz=nz, density=density, substeps=substeps, every=every)
    return dict(c, name=name) if name else c


def _scene_grad(name, material, nx, ny, nz, density, steps, substeps):
    c = dict(kind="scene_grad", material=material, nx=nx, ny=ny, nz=nz, density=density, steps=steps, substeps=substeps)
    return dict(c, name=name) if name else c


def _sdf(name, res, around, along):
    c = dict(kind="sdf", res=res, around=around, along=along)
    return dict(c, name=name) if name else c


def listed():
    return [
        # a control loop around one small soft body: the latency of a step is all there is
        _scene("control_1k", "elastic", 10, 10, 10, 64, 2, 10),
        # the single elastic cube of the README, one hundred substeps of a recorded clip
        _scene("cube_32k", "elastic", 32, 32, 32, 64, 4, 25),
        # reinforcement learning: copies of one actuated muscle body, a new action every step
        _scene("muscle_envs", "muscle", 12, 10, 17, 64, 4, 10, envs=16),
        # granular material poured over a fixed sphere (coupled grid op), sizes that fill no block evenly
        _scene("sand_sphere", "sand", 47, 41, 29, 96, 1, 50, sphere=True),
        # the benchmark scene: four materials, 500,000 particles, one hundred substeps
        _scene("mixed_500k", "mixed", 50, 50, 50, 128, 1, 100),
        # an offline-quality simulation, the state streams from HBM
        _scene("mixed_4m", "mixed", 100, 100, 100, 256, 1, 20),
        # parameter study: uneven scenes of every material and grid advanced together
        _batch("batch_40", 40, 2000, 60000, 100),
        # system identification: gradients of a rollout w.r.t. initial velocities and per-particle E
        _grad("grad_20k", "elastic", 25, 25, 32, 64, 200, 20),
        # the same for a small plastic body, with an odd number of substeps
        _grad("grad_sand_3k", "sand", 13, 17, 14, 64, 75, 20),
        # trajectory optimisation through a differentiable scene, a loss on the last state
        _scene_grad("scene_grad_4k", "neohooken", 16, 16, 16, 64, 6, 10),
        # building a scene with a tool: its mesh's signed-distance grid
        _sdf("tool_sdf", 96, 40, 17),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _lattice(rng, n, most):
    """Three uneven edges whose product is about n, none above most."""
    a = min(most, max(3, round(n ** (1 / 3) * rng.uniform(0.7, 1.4))))
    b = min(most, max(3, round(math.sqrt(n / a) * rng.uniform(0.8, 1.25))))
    return a, b, min(most, max(3, round(n / (a * b))))


def draw(rng):
    kind = rng.choice(("scene",) * 8 + ("mixed",) * 3 + ("batch",) * 3 + ("grad",) * 3 + ("scene_grad", "sdf"))
    if kind == "scene":
        material = rng.choice(("elastic", "neohooken", "liquid", "sand", "snow", "elastoplastic", "muscle"))
        density = rng.choice((32, 48, 64, 96, 128))
        n = _log(rng, 500, 400e3)
        sphere = rng.random() < 0.25
        nx, ny, nz = _lattice(rng, n, int((0.5 if sphere else 0.8) * 2 * density))
        envs = 0 if n > 20e3 or rng.random() < 0.6 else round(_log(rng, 2, 40))
        steps = rng.choice((1, 1, 2, 3, 5))
        top = min(120, 4e7 / (nx * ny * nz * max(envs, 1)))
        return _scene(None, material, nx, ny, nz, density, steps, max(2, round(_log(rng, 4, max(5, top)) / steps)), envs,
                      sphere)
    if kind == "mixed":
        density = rng.choice((64, 96, 128, 160, 192))
        side = min(round(_log(rng, 8, 90)), int(0.6 * density))
        return _scene(None, "mixed", side, max(4, side - rng.randrange(3)), max(4, side - rng.randrange(5)), density, 1,
                      max(4, round(_log(rng, 6, min(120, 4e7 / (4 * side**3))))))
    if kind == "batch":
        lo = round(_log(rng, 500, 5000))
        hi = round(lo * rng.uniform(1, 25))
        return _batch(None, round(_log(rng, 3, 60)), lo, hi, round(_log(rng, 10, 120)))
    if kind == "grad":
        material = rng.choice(("elastic", "neohooken", "liquid", "sand", "snow", "elastoplastic"))
        density = rng.choice((48, 64, 96))
        nx, ny, nz = _lattice(rng, _log(rng, 600, 40e3), 60)
        return _grad(None, material, nx, ny, nz, density, round(_log(rng, 20, 150)), rng.choice((10, 20, 25)))
    if kind == "scene_grad":
        nx, ny, nz = _lattice(rng, _log(rng, 600, 12e3), 40)
        return _scene_grad(None, rng.choice(("elastic", "neohooken", "liquid")), nx, ny, nz, 64, rng.randint(2, 6),
                           rng.choice((5, 10, 20)))
    return _sdf(None, round(_log(rng, 24, 128)), rng.randint(8, 50), rng.randint(5, 24))


# ---------------------------------------------------------------- inputs


def _materials(case):
    return MIXED if case["material"] == "mixed" else (case["material"],)


def _geometry(case):
    """Per material: the lower corner and the particle spacing of its block."""
    dx = 1.0 / case["density"]
    dims = (case["nx"], case["ny"], case["nz"])
    if case["material"] == "mixed":  # four blocks, one per xy quadrant, at different heights
        h = 0.64 * dx
        q = (1.0 - 8 * dx) / 2
        return [(tuple(4 * dx + (m, k)[a] * q + (q - dims[a] * h) / 2 for a in (0, 1)) + (4 * dx + 0.05 * (m + 2 * k),), h)
                for k in (0, 1) for m in (0, 1)]
    h = 0.5 * dx
    z = 0.32 if case.get("sphere") else 3.4 * dx
    return [((0.5 - dims[0] * h / 2, 0.5 - dims[1] * h / 2, z), h)]


def _inputs(case, seed):
    """float32 state on the GPU, [envs, n, ...]: blocks in motion with F around the identity."""
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    B = max(1, case.get("envs", 0))
    axes = [torch.arange(case[k], device=DEV, dtype=torch.float64) + 0.5 for k in ("nx", "ny", "nz")]
    lat = torch.stack(torch.meshgrid(*axes, indexing="ij"), -1).reshape(-1, 3)
    parts = [torch.tensor(lo, device=DEV, dtype=torch.float64) + lat * h for lo, h in _geometry(case)]
    h = _geometry(case)[0][1]
    base = torch.cat(parts)
    n = len(base)

    def noise(*shape):
        return torch.randn(shape, generator=g, device=DEV, dtype=torch.float32)

    jitter = torch.rand((B, n, 3), generator=g, device=DEV, dtype=torch.float64) - 0.5
    pos = (base + 0.5 * h * jitter).float()
    vel = torch.tensor([0.4, -0.2, -1.5], device=DEV) + 0.2 * noise(B, n, 3)
    F = torch.eye(3, device=DEV) + 0.01 * noise(B, n, 3, 3)
    jp = torch.ones((B, n), device=DEV)
    mats = _materials(case)
    for k, m in enumerate(mats):
        if m == "sand":
            jp[:, k * len(lat):(k + 1) * len(lat)] = 0.0
    s = dict(pos=pos, vel=vel, C=2.0 * noise(B, n, 3, 3), F=F, Jp=jp)
    if case["material"] == "muscle":
        s["actu"] = 0.5 * torch.rand((case["steps"], B, 1), generator=g, device=DEV)
    return s


def _substep_dt(density):
    return 6.4e-3 / density


def _gs_material(name):
    from genesis_b200.materials import MPM

    E = YOUNG[name]
    if name in ("elastic", "neohooken"):
        return MPM.Elastic(E=E, nu=NU, rho=RHO, model="corotation" if name == "elastic" else "neohooken")
    if name == "muscle":
        return MPM.Muscle(E=E, nu=NU, rho=RHO)
    if name == "snow":
        return MPM.Snow(E=E, nu=NU, rho=RHO, yield_lower=2.5e-2, yield_higher=7.5e-3)
    cls = {"liquid": MPM.Liquid, "sand": MPM.Sand, "elastoplastic": MPM.ElastoPlastic}[name]
    return cls(E=E, nu=NU, rho=RHO)


def _build_scene(case, requires_grad=False):
    import genesis_b200 as gs

    gs.init(backend=gs.gpu, precision="32", seed=0, logging_level="error")
    (_, h) = _geometry(case)[0]
    S = case["substeps"]
    scene = gs.Scene(
        sim_options=gs.options.SimOptions(dt=_substep_dt(case["density"]) * S, substeps=S, gravity=(0.0, 0.0, -9.8),
                                          requires_grad=requires_grad),
        mpm_options=gs.options.MPMOptions(lower_bound=(0, 0, 0), upper_bound=(1, 1, 1), grid_density=case["density"],
                                          particle_size=h),
    )
    if case.get("sphere"):
        scene.add_entity(gs.morphs.Sphere(pos=(0.5, 0.5, 0.2), radius=0.12),
                         material=gs.materials.Rigid(coup_friction=0.3))
    dims = np.array([case["nx"], case["ny"], case["nz"]])
    ents = []
    for (lo, h), m in zip(_geometry(case), _materials(case)):
        mat = _gs_material(m)
        mat._sampler = "regular"  # the lattice: one particle per cell of the morph
        ents.append(scene.add_entity(gs.morphs.Box(lower=lo, upper=tuple(np.array(lo) + dims * h)), material=mat))
    scene.build(n_envs=case.get("envs", 0))
    return scene, ents


def _desc(case, s, seed_E=None):
    from genesis_b200.workloads import SceneDesc

    name = case["material"]
    kw = dict(E=YOUNG[name], nu=NU, rho=RHO)
    kind = name
    if name == "neohooken":
        kind, kw = "elastic", dict(kw, model="neohooken")
    if name == "snow":
        kw = dict(kw, yield_lower=2.5e-2, yield_higher=7.5e-3)
    n = s["pos"].shape[1]
    return SceneDesc(name=name, grid_density=case["density"], particle_size=_geometry(case)[0][1],
                     dt=_substep_dt(case["density"]), n_substeps=case["substeps"],
                     pos=s["pos"][0].cpu().numpy().astype(np.float64), vel=s["vel"][0].cpu().numpy().astype(np.float64),
                     mat_idx=np.zeros(n, dtype=np.int64), materials=[(kind, kw)], E_particle=seed_E)


def _batch_scenes(case):
    """Sizes spread over [n_lo, n_hi], grids and materials cycling."""
    out = []
    for i in range(case["scenes"]):
        t = ((i * 0.618034) % 1.0) if case["scenes"] > 1 else 0.5
        n = case["n_lo"] * (case["n_hi"] / case["n_lo"]) ** t
        density = (32, 64, 96)[i % 3]
        a = min(max(3, round(n ** (1 / 3))), 2 * density - 24)
        c = min(max(3, round(n / (a * a))), 2 * density - 24)
        out.append(dict(material=("elastic", "liquid", "sand", "snow", "elastoplastic")[i % 5], nx=a, ny=a, nz=c,
                        density=density, substeps=case["substeps"]))
    return out


def _youngs(case, seed):
    n = case["nx"] * case["ny"] * case["nz"]
    g = torch.Generator(device=DEV).manual_seed(int(seed) + 17)
    return YOUNG[case["material"]] * torch.exp(0.3 * torch.randn(n, generator=g, device=DEV))


_GOAL = (0.55, 0.5, 0.25)


def _bumpy_sphere(case, seed):
    """A closed latitude-longitude mesh of unit extent with a few seeded bumps."""
    nu, nv = case["around"], case["along"]
    r = np.random.default_rng(seed)
    k, ph = r.integers(1, 5, size=(4, 2)), r.uniform(0, 2 * math.pi, size=(4, 2))
    th = np.pi * np.arange(1, nv) / nv
    al = 2 * np.pi * np.arange(nu) / nu
    T, A = np.meshgrid(th, al, indexing="ij")
    rad = 0.4 + sum(0.015 * np.sin(a * T + p) * np.cos(b * A + q) * np.sin(T) for (a, b), (p, q) in zip(k, ph))
    ring = np.stack([rad * np.sin(T) * np.cos(A), rad * np.sin(T) * np.sin(A), rad * np.cos(T)], -1).reshape(-1, 3)
    v = np.concatenate([ring, [[0, 0, 0.4], [0, 0, -0.4]]])
    top, bot = len(ring), len(ring) + 1
    f = []
    for j in range(nu):
        m = (j + 1) % nu
        f.append((top, j, m))
        f.append((bot, (nv - 2) * nu + m, (nv - 2) * nu + j))
        for i in range(nv - 2):
            a, b, c, d = i * nu + j, i * nu + m, (i + 1) * nu + j, (i + 1) * nu + m
            f += [(a, c, b), (b, c, d)]
    return v, np.array(f, dtype=np.int32)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "scene":
        from genesis_b200.engine.states import MPMSolverState

        scene, ents = _build_scene(case)
        s = _inputs(case, seed)
        active = torch.ones(s["pos"].shape[:2], dtype=torch.bool, device=DEV)
        state = MPMSolverState(scene, s["pos"], s["vel"], s["C"], s["F"], s["Jp"], active)
        return dict(case=case, scene=scene, ents=ents, state=state, actu=s.get("actu"))
    if kind == "batch":
        from genesis_b200.batch import BatchedScenes

        descs, parts = [], []
        for i, sc in enumerate(_batch_scenes(case)):
            s = _inputs(sc, seed * 1009 + i)
            parts.append(s)
            descs.append(_desc(sc, s))
        # 256-particle work items re-sorted every 100 substeps: what the tuner picks for batches
        sim = BatchedScenes(descs, tune=False, chunk_particles=256, sort_interval=100)
        cat = {k: torch.cat([p[k][0] for p in parts]) for k in ("pos", "vel", "C", "F", "Jp")}
        return dict(case=case, sim=sim, **cat)
    if kind == "grad":
        from genesis_b200.grad import DifferentiableRollout

        s = _inputs(case, seed)
        E = _youngs(case, seed)
        sim = DifferentiableRollout(_desc(case, s, E.cpu().numpy().astype(np.float64)), checkpoint_every=case["every"])
        return dict(case=case, sim=sim, v0=s["vel"][0].clone().requires_grad_(), E=E.clone().requires_grad_(),
                    goal=torch.tensor(_GOAL, device=DEV))
    if kind == "scene_grad":
        scene, ents = _build_scene(case, requires_grad=True)
        s = _inputs(case, seed)
        return dict(case=case, scene=scene, ent=ents[0], pos=s["pos"][0].clone().requires_grad_(),
                    vel=s["vel"][0].clone().requires_grad_(), goal=torch.tensor(_GOAL, device=DEV))
    v, f = _bumpy_sphere(case, seed)
    return dict(case=case, v=v, f=f)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "scene":
        scene = state["scene"]
        scene.reset(state["state"])
        for k in range(case["steps"]):
            if state["actu"] is not None:
                state["ents"][0].set_actuation(state["actu"][k])
            scene.step()
        st = scene.get_state()[3]
        return dict(pos=st.pos, vel=st.vel, C=st.C, F=st.F, Jp=st.Jp, active=st.active)
    if kind == "batch":
        sim = state["sim"]
        sim.rt.set_state(pos=state["pos"], vel=state["vel"], C_=state["C"], F=state["F"], Jp=state["Jp"])
        sim.substeps(case["substeps"])
        return sim.rt.get_state()
    if kind == "grad":
        from genesis_b200.grad import rollout

        state["v0"].grad = state["E"].grad = None
        x = rollout(state["v0"], state["E"], state["sim"])
        ((x - state["goal"]) ** 2).sum(-1).mean().backward()
        return dict(pos=x.detach(), v0=state["v0"].grad, E=state["E"].grad)
    if kind == "scene_grad":
        scene = state["scene"]
        state["pos"].grad = state["vel"].grad = None
        scene.reset()
        state["ent"].set_position(state["pos"])
        state["ent"].set_velocity(state["vel"])
        for _ in range(case["steps"]):
            scene.step()
        st = scene.get_state()[3]
        ((st.pos[0] - state["goal"]) ** 2).sum(-1).mean().backward()
        return dict(pos=st.pos.detach(), x0=state["pos"].grad, v0=state["vel"].grad)
    from genesis_b200.engine.tool import sdf_voxels

    return sdf_voxels(state["v"], state["f"], case["res"], DEV)


def work(case):
    """Bytes: the particle state in and out of every substep (208 B with its share of the
    grid; a gradient walks the substeps forward and back).  Operations: about 1,500 per particle
    and substep (27-node gather and scatter, SVD, return mapping), twice that in reverse."""
    kind = case["kind"]
    if kind == "sdf":
        faces = 2 * case["around"] * (case["along"] - 1)
        # each node: the distance to the few triangles near it, and its sign
        return {"bytes": 4.0 * case["res"] ** 3 + 24.0 * faces, "flops": 2000.0 * case["res"] ** 3}
    if kind == "batch":
        n = sum(s["nx"] * s["ny"] * s["nz"] for s in _batch_scenes(case)) * case["substeps"]
    else:
        n = case["nx"] * case["ny"] * case["nz"] * len(_materials(case)) * max(1, case.get("envs", 0))
        n *= case["substeps"] * case.get("steps", 1)
    k = 3 if kind in ("grad", "scene_grad") else 1
    return {"bytes": 208.0 * n * k, "flops": 1500.0 * n * k}


# ---------------------------------------------------------------- float64 restatement


def _jacobi_svd(F):
    """U, s, V of [n, 3, 3] well-conditioned matrices (cyclic Jacobi on F^T F)."""
    A = F.transpose(1, 2) @ F
    a = {(i, j): A[:, i, j].clone() for i in range(3) for j in range(i, 3)}
    one, zero = torch.ones_like(a[0, 0]), torch.zeros_like(a[0, 0])
    v = [[one.clone() if i == j else zero.clone() for j in range(3)] for i in range(3)]
    for _ in range(5):
        for p, q in ((0, 1), (0, 2), (1, 2)):
            r = 3 - p - q
            apq = a[p, q]
            d = a[q, q] - a[p, p]
            e = 2 * apq
            den = d.abs() + torch.sqrt(d * d + e * e)
            t = torch.where(den > 0, e / torch.where(den > 0, den, one), zero) * torch.where(d < 0, -one, one)
            c = torch.rsqrt(1 + t * t)
            s = t * c
            a[p, p], a[q, q], a[p, q] = a[p, p] - t * apq, a[q, q] + t * apq, zero
            kp, kq = (min(r, p), max(r, p)), (min(r, q), max(r, q))
            a[kp], a[kq] = c * a[kp] - s * a[kq], s * a[kp] + c * a[kq]
            for i in range(3):
                v[i][p], v[i][q] = c * v[i][p] - s * v[i][q], s * v[i][p] + c * v[i][q]
    V = torch.stack([torch.stack(row, -1) for row in v], 1)
    s = torch.sqrt(torch.stack([a[k, k] for k in range(3)], -1))
    return (F @ V) / s[:, None, :], s, V


def _inverse_transpose(F):
    K = torch.stack([torch.linalg.cross(F[:, 1], F[:, 2]), torch.linalg.cross(F[:, 2], F[:, 0]),
                     torch.linalg.cross(F[:, 0], F[:, 1])], 1)
    return K / (F[:, 0] * K[:, 0]).sum(-1)[:, None, None]


def _rotation(F):
    """The polar rotation (Newton iteration, differentiable)."""
    R = F
    for _ in range(6):
        R = 0.5 * (R + _inverse_transpose(R))
    return R


def _constitutive(name, Ft, Jp, mu, lam, actu):
    """(F_new, Jp_new, stress) of one material; mu, lam numbers or [n] tensors."""
    eye = torch.eye(3, dtype=Ft.dtype, device=Ft.device)

    def col(x):
        return x[:, None, None] if torch.is_tensor(x) and x.ndim == 1 else x

    J = (Ft[:, 0] * torch.linalg.cross(Ft[:, 1], Ft[:, 2])).sum(-1)
    if name == "liquid":
        Fn = J.clamp_min(0).pow(1 / 3)[:, None, None] * eye
        return Fn, Jp, col(lam * J * (J - 1)) * eye
    if name in ("neohooken", "muscle"):
        P = col(mu) * (Ft @ Ft.transpose(1, 2)) + col(lam * torch.log(J) - mu) * eye
        if actu is not None:
            g = Ft[:, :, 2]  # the default fibre direction, z
            P = P + (YOUNG["muscle"] * actu)[:, None, None] * g[:, :, None] * g[:, None, :]
        return Ft, Jp, P
    if name == "elastic":
        P = 2 * col(mu) * ((Ft - _rotation(Ft)) @ Ft.transpose(1, 2)) + col(lam * J * (J - 1)) * eye
        return Ft, Jp, P
    U, s, V = _jacobi_svd(Ft)

    def spectral(d, W):
        return (U * d[:, None, :]) @ W.transpose(1, 2)

    if name == "sand":
        sin_phi = math.sin(math.radians(45))
        alpha = math.sqrt(2 / 3) * 2 * sin_phi / (3 - sin_phi)
        e = torch.log(s.clamp_min(1e-4))
        tr = e.sum(-1) + Jp
        eh = e - (tr / 3)[:, None]
        nn = torch.sqrt((eh * eh).sum(-1) + EPS)
        dg = (nn + (3 * lam + 2 * mu) / (2 * mu) * tr * alpha).clamp_min(0)
        out = tr >= 0
        ls = torch.where(out[:, None], torch.zeros_like(e), e - (dg / nn)[:, None] * eh)
        lam_c = lam[:, None] if torch.is_tensor(lam) else lam
        mu_c = mu[:, None] if torch.is_tensor(mu) else mu
        P = spectral(2 * mu_c * ls + lam_c * ls.sum(-1, keepdim=True), U)
        return spectral(torch.exp(ls), V), torch.where(out, tr, torch.zeros_like(tr)), P
    if name == "snow":
        sn = s.clamp(1 - 2.5e-2, 1 + 7.5e-3)
        Jn = Jp * (s / sn).prod(-1)
        h = torch.exp(10 * (1 - Jp))
        mu, lam = mu * h, lam * h
    else:  # von Mises
        e = torch.log(s.clamp_min(0.05))
        eh = e - e.mean(-1, keepdim=True)
        nn = torch.sqrt((eh * eh).sum(-1) + EPS)
        mu0 = YOUNG[name] / (2 * (1 + NU))
        dg = nn - 1e4 / (2 * mu0) * (mu0 / mu)
        sn = torch.where((dg > 0)[:, None], torch.exp(e - (dg / nn)[:, None] * eh), s)
        Jn = Jp
    mu_c = mu[:, None] if torch.is_tensor(mu) else mu
    P = spectral(2 * mu_c * (sn - 1) * sn, U) + col(lam * J * (J - 1)) * eye
    return spectral(sn, V), Jn, P


def _sphere_response(pos, v):
    """A fixed sphere of radius 0.12 at (0.5, 0.5, 0.2), friction 0.3, softness 0.002."""
    q = pos - torch.tensor([0.5, 0.5, 0.2], dtype=pos.dtype, device=pos.device)
    r = torch.sqrt((q * q).sum(-1))
    infl = torch.exp(-(r - 0.12) / 0.002).clamp_max(1.0)
    n = q / torch.sqrt((q * q).sum(-1, keepdim=True) + EPS)
    n = n / torch.sqrt((n * n).sum(-1, keepdim=True) + EPS)
    rn = (v * n).sum(-1, keepdim=True)
    rt = v - rn * n
    m = torch.sqrt((rt * rt).sum(-1, keepdim=True) + EPS)
    new = rt * (m + rn * 0.3).clamp_min(0) / m
    i = infl[:, None]
    return torch.where((i > 0.1) & (rn < 0), new * i + v * (1 - i), v)


def _exact_steps(case, s, mats, substeps, E=None, sphere=False):
    """Advance the float64 state s of [envs, n, ...] tensors; mats: (material, particles) in
    order; substeps: a list of the actuation ([envs, 1] or None) of every substep."""
    density = case["density"]
    dt, dx, inv = _substep_dt(density), 1.0 / density, float(density)
    B, n = s["pos"].shape[:2]
    x, v, C, F, Jp = (s[k].reshape((B * n,) + s[k].shape[2:]) for k in ("pos", "vel", "C", "F", "Jp"))
    h = _geometry(case)[0][1]
    vol = h**3 * 1e3
    mass = vol * RHO
    res = density + 1
    env = torch.arange(B, device=x.device).repeat_interleave(n) * res**3
    lo, hi = 3 * dx, 1 - 3 * dx
    ends = np.cumsum([0] + [k for _, k in mats])
    local = torch.arange(B * n, device=x.device) % n
    node = torch.stack(torch.meshgrid(*[torch.arange(res, device=x.device)] * 3, indexing="ij"), -1).reshape(-1, 3)
    gpos = (node.to(x.dtype) * dx).repeat(B, 1)
    for a in substeps:
        Ft = F + dt * (C @ F)
        actu = None if a is None else a.to(x.dtype).expand(B, n).reshape(-1)
        Fn, Jn, P = [], [], []
        sel = [slice(None)] if len(mats) == 1 else [(local >= ends[k]) & (local < ends[k + 1]) for k in range(len(mats))]
        for (name, _), i in zip(mats, sel):
            e = YOUNG[name] if E is None else E
            mu, lam = e / (2 * (1 + NU)), e * NU / ((1 + NU) * (1 - 2 * NU))
            f, j, p = _constitutive(name, Ft[i], Jp[i], mu, lam, actu)
            Fn.append(f), Jn.append(j), P.append(p)
        if len(mats) == 1:
            F, Jp, P = Fn[0], Jn[0], P[0]
        else:
            out = [torch.empty_like(Ft), torch.empty_like(Jp), torch.empty_like(Ft)]
            for k, i in enumerate(sel):
                out[0][i], out[1][i], out[2][i] = Fn[k], Jn[k], P[k]
            F, Jp, P = out
        A = -dt * vol * 4 * inv * inv * P + mass * C
        base = torch.floor(x.detach() * inv - 0.5)
        fx = x * inv - base
        w = [0.5 * (1.5 - fx) ** 2, 0.75 - (fx - 1) ** 2, 0.5 * (fx - 0.5) ** 2]
        b = base.long()
        grid = torch.zeros((B * res**3, 4), dtype=x.dtype, device=x.device)
        nodes = []
        for i in range(3):
            for j in range(3):
                for k in range(3):
                    off = torch.tensor([i, j, k], dtype=x.dtype, device=x.device) - fx
                    wt = w[i][:, 0] * w[j][:, 1] * w[k][:, 2]
                    idx = env + ((b[:, 0] + i) * res + b[:, 1] + j) * res + b[:, 2] + k
                    nodes.append((idx, wt, off))
                    mom = mass * v + (A @ (off * dx)[:, :, None])[:, :, 0]
                    grid = grid.index_add(0, idx, torch.cat([wt[:, None] * mom, (wt * mass)[:, None]], 1)) \
                        if grid.requires_grad or mom.requires_grad else \
                        grid.index_add_(0, idx, torch.cat([wt[:, None] * mom, (wt * mass)[:, None]], 1))
                    if not torch.is_grad_enabled():
                        nodes[-1] = (i, j, k)
        m = grid[:, 3:]
        live = m > EPS
        gv = torch.where(live, grid[:, :3] / torch.where(live, m, torch.ones_like(m)), torch.zeros_like(m))
        gv = torch.where(live, gv + dt * torch.tensor([0.0, 0.0, -9.8], dtype=x.dtype, device=x.device), gv)
        if sphere:
            gv = torch.where(live, _sphere_response(gpos, gv), gv)
        stop = ((gpos >= hi - 1e-9) & (gv >= 0)) | ((gpos <= lo + 1e-9) & (gv <= 0))
        gv = torch.where(stop, torch.zeros_like(gv), gv)
        nv, nC = 0.0, 0.0
        for item in nodes:
            if torch.is_tensor(item[0]):
                idx, wt, off = item
            else:
                i, j, k = item
                off = torch.tensor([i, j, k], dtype=x.dtype, device=x.device) - fx
                wt = w[i][:, 0] * w[j][:, 1] * w[k][:, 2]
                idx = env + ((b[:, 0] + i) * res + b[:, 1] + j) * res + b[:, 2] + k
            g = wt[:, None] * gv[idx]
            nv = nv + g
            nC = nC + 4 * inv * g[:, :, None] * off[:, None, :]
        nx = x + dt * nv
        stop = ((nx >= hi) & (nv >= 0)) | ((nx <= lo) & (nv <= 0))
        v, C, x = torch.where(stop, torch.zeros_like(nv), nv), nC, nx.clamp(lo, hi)
    shape = {"pos": x, "vel": v, "C": C, "F": F, "Jp": Jp}
    return {k: t.reshape((B, n) + t.shape[1:]) for k, t in shape.items()}


def _double(s):
    return {k: t.double() for k, t in s.items()}


def _exact_gradient(case, s, E, total):
    n = s["pos"].shape[1]
    s["C"] = torch.zeros_like(s["C"])
    s["F"] = torch.eye(3, dtype=torch.float64, device=DEV).expand(1, n, 3, 3).clone()
    smooth = case["material"] in ("elastic", "neohooken", "liquid")
    leaves = {"x0": s["pos"], "v0": s["vel"]}
    if E is not None:
        leaves["E"] = E
    if smooth:
        leaves = {k: t.clone().requires_grad_() for k, t in leaves.items()}
        s = dict(s, pos=leaves["x0"], vel=leaves["v0"])
    with torch.set_grad_enabled(smooth):
        out = _exact_steps(case, s, [(case["material"], n)], [None] * total, E=leaves.get("E"))
        goal = torch.tensor(_GOAL, device=DEV).double()
        if smooth:
            ((out["pos"][0] - goal) ** 2).sum(-1).mean().backward()
    return out["pos"].detach(), {k: t.grad if smooth else None for k, t in leaves.items()}


def _exact_sdf(v, f, res):
    v = torch.as_tensor(v.astype(np.float32), device=DEV).double()
    tri = v[torch.as_tensor(f, device=DEV).long()]
    ax = torch.linspace(-0.6, 0.6, res, dtype=torch.float64, device=DEV)
    p = torch.stack(torch.meshgrid(ax, ax, ax, indexing="ij"), -1).reshape(-1, 3)
    out = torch.empty(len(p), dtype=torch.float64, device=DEV)
    a, b, c = tri[:, 0], tri[:, 1], tri[:, 2]
    nrm = torch.linalg.cross(b - a, c - a)
    unit = nrm / nrm.norm(dim=-1, keepdim=True)
    step = max(1, 24_000_000 // len(tri))

    def dot(x, y):
        return (x * y).sum(-1)

    for i in range(0, len(p), step):
        q = p[i:i + step][:, None, :]
        best, inside = None, None
        for s, e in ((a, b), (b, c), (c, a)):
            d = e - s
            t = (dot(q - s, d) / dot(d, d)).clamp(0, 1)
            g = q - s - t[..., None] * d
            d2 = dot(g, g)
            best = d2 if best is None else torch.minimum(best, d2)
            side = dot(torch.linalg.cross(d, unit)[None], q - s) <= 0  # inside of this edge
            inside = side if inside is None else inside & side
            del g, d2, t, side
        h = dot(q - a, unit)
        d2 = torch.where(inside, h * h, best).amin(1)
        ra, rb, rc = a - q, b - q, c - q
        la, lb, lc = ra.norm(dim=-1), rb.norm(dim=-1), rc.norm(dim=-1)
        det = dot(ra, torch.linalg.cross(rb, rc))
        den = la * lb * lc + dot(ra, rb) * lc + dot(ra, rc) * lb + dot(rb, rc) * la
        w = 2 * torch.atan2(det, den).sum(1) / (4 * math.pi)
        out[i:i + step] = torch.where(w.abs() > 0.5, -1.0, 1.0) * torch.sqrt(d2)
    return out.reshape(res, res, res)


def exact(case, seed):
    kind = case["kind"]
    if kind == "sdf":
        v, f = _bumpy_sphere(case, seed)
        return _exact_sdf(v, f, case["res"])
    if kind == "scene":
        s = _double(_inputs(case, seed))
        n = case["nx"] * case["ny"] * case["nz"]
        acts = [s["actu"][k] if "actu" in s else None for k in range(case["steps"]) for _ in range(case["substeps"])]
        with torch.no_grad():
            out = _exact_steps(case, s, [(m, n) for m in _materials(case)], acts, sphere=case["sphere"])
        return dict(out, active=None)
    if kind == "batch":
        outs = []
        for i, sc in enumerate(_batch_scenes(case)):
            s = _double(_inputs(sc, seed * 1009 + i))
            with torch.no_grad():
                outs.append(_exact_steps(sc, s, [(sc["material"], s["pos"].shape[1])], [None] * sc["substeps"]))
        return dict({k: torch.cat([o[k][0] for o in outs]) for k in ("pos", "vel", "C", "F", "Jp")}, active=None)
    s = _double(_inputs(case, seed))
    if kind == "grad":
        pos, g = _exact_gradient(case, s, _youngs(case, seed).double(), case["substeps"])
        return dict(pos=pos[0], v0=None if g["v0"] is None else g["v0"][0], E=g["E"])
    pos, g = _exact_gradient(case, s, None, case["steps"] * case["substeps"])
    return dict(pos=pos, x0=g["x0"][0], v0=g["v0"][0])
