"""The recorded reverse pass against the float64 adjoint, substep by substep along the states that
the GPU itself recorded.

Along a rollout the plastic return mappings switch branch (and their derivatives jump) where the
states of two runs differ by a rounding, so whole gradients are reproducible to no more than that.
Here both sides differentiate the same recorded state: a particle within MARGIN of a switch (a yield
or expansion surface, a clamp, or two singular values that the float64 form treats as one), which
float32 may put on the other side, is left out of the material's outputs (C, F, Jp, mu, lam; the
adjoints of x and v are formed before the material); the block hangs free of the walls.

Tolerances, of the 2-norm of each channel group: with the singular values perturbed by 2e-7 and
F_tmp, the node velocities and the momentum by one float32 rounding, the float64 adjoint of these
scenes moves by at most 2e-7 (x), 4.5e-5 (C, F), 1.2e-4 (Jp) and 2.7e-4 (mu, lam); four times that is
allowed, and 2e-5 for x and v, whose float32 sums over 27 nodes and up to 64 particles a node are what
they consist of."""

import ctypes as C

import numpy as np
import pytest
import torch

from genesis_b200 import _native as nat
from genesis_b200 import workloads as W

MATERIALS = [
    ("elastic", dict(E=1e5, nu=0.3)),
    ("elastoplastic", dict(E=1e5, nu=0.3, von_mises_yield_stress=2e3)),
    ("elastoplastic", dict(E=1e5, nu=0.3, use_von_mises=False)),
    ("liquid", dict(E=1e5, nu=0.2, viscous=True)),
    ("sand", dict(E=1e5, friction_angle=40)),
    ("snow", dict(E=1e5, yield_lower=2.5e-2, yield_higher=7.5e-3)),
]
GROUPS = {"x": slice(0, 3), "v": slice(3, 6), "C": slice(6, 15), "F": slice(15, 24), "Jp": slice(24, 25)}
TOL = {"x": 2e-5, "v": 2e-5, "C": 1.8e-4, "F": 1.8e-4, "Jp": 4.8e-4, "mu": 1.1e-3, "lam": 1.1e-3}
MARGIN = 1e-5
STRAIN = 2e-2


def _desc(kind, kw, side, T, seed=11):
    rng = np.random.default_rng(seed)
    dx = 1.0 / 32
    pos = W.jittered_lattice(rng, side, (0.28, 0.26, 0.3), 0.5 * dx)
    n = len(pos)
    return W.SceneDesc(name="records", grid_density=32, particle_size=0.5 * dx, dt=2e-4, n_substeps=T, pos=pos,
                       vel=rng.normal(0.0, 0.5, size=(n, 3)), mat_idx=np.zeros(n, dtype=np.int64),
                       materials=[(kind, dict(kw))], upper_bound=(1.0, 1.0, 1.0),
                       E_particle=kw["E"] * np.exp(0.5 * rng.normal(size=n)))


def _state(d, kind, seed=12):
    """Strained particles in motion: F = I + N(0, STRAIN), C ~ N(0, 10 / s), Jp off its default."""
    rng = np.random.default_rng(seed)
    n = d.n_particles
    F = np.eye(3) + rng.normal(0.0, STRAIN, size=(n, 3, 3))
    jp = {"snow": 1.0 + 0.02 * rng.normal(size=n), "sand": -0.03 * np.abs(rng.normal(size=n))}.get(kind, np.zeros(n))
    return F, rng.normal(0.0, 10.0, size=(n, 3, 3)), jp


def _lame(d):
    nu = d.materials[0][1].get("nu", 0.2)
    E = d.E_particle
    return E / (2 * (1 + nu)), E * nu / ((1 + nu) * (1 - 2 * nu))


def _seed_adjoint(n, seed=13):
    """An output adjoint whose channels weigh about the same in the input's: those of a loss on x."""
    rng = np.random.default_rng(seed)
    a = rng.normal(size=(nat.MPM_STATE_CH, n))
    a[GROUPS["v"]] *= 1e-2
    a[GROUPS["C"]] *= 1e-4
    return a


def _clear(mat, eps, S, Jp, mu, lam):
    """Particles whose material is MARGIN away from every switch."""
    from oracle import mpm_ref as R

    gap = np.full(len(S), np.inf)
    for i, j in ((0, 1), (1, 2), (0, 2)):
        gap = np.minimum(gap, np.abs(S[:, i] ** 2 - S[:, j] ** 2) - 1e-6)  # the float64 form's guard
    if mat.kind == R.KIND_ELASTOPLASTIC and mat.use_von_mises:
        e = np.log(np.maximum(S, 0.05))
        eh = e - e.mean(1, keepdims=True)
        gap = np.minimum(gap, np.abs(np.sqrt((eh * eh).sum(1) + eps) - mat.von_mises_yield_stress / (2 * mu)))
    elif mat.kind in (R.KIND_ELASTOPLASTIC, R.KIND_SNOW):
        for edge in (1 - mat.yield_lower, 1 + mat.yield_higher):
            gap = np.minimum(gap, np.abs(S - edge).min(1))
    elif mat.kind == R.KIND_SAND:
        e = np.log(S)
        tr = e.sum(1) + Jp
        eh = e - (tr / 3)[:, None]
        nn = np.sqrt((eh * eh).sum(1) + eps)
        gap = np.minimum(gap, np.minimum(np.abs(tr), np.abs(nn + (3 * lam + 2 * mu) / (2 * mu) * tr * mat.alpha)))
    return gap > MARGIN


def _oracle_state(chan, mu, lam):
    a = np.asarray(chan, dtype=np.float64)
    n = a.shape[1]
    st = dict(x=a[0:3].T.copy(), v=a[3:6].T.copy(), C=a[6:15].T.reshape(n, 3, 3).copy(),
              F=a[15:24].T.reshape(n, 3, 3).copy(), Jp=a[24].copy(), mat=np.zeros(n, dtype=np.int64))
    return st, np.asarray(mu, dtype=np.float64), np.asarray(lam, dtype=np.float64)


def _oracle_adjoint(p, mats, st, mu, lam, out):
    """The adjoint of the input state [25, n], of mu and lam, and the particles clear of a switch."""
    from oracle import mpm_adjoint as A

    n = len(mu)
    adj = dict(x=out[0:3].T, v=out[3:6].T, C=out[6:15].T.reshape(n, 3, 3), F=out[15:24].T.reshape(n, 3, 3), Jp=out[24])
    _, inter = A.forward_materials(p, mats, st, mu, lam)
    a, mb, lb, _ = A.backward_materials(p, mats, st, mu, lam, inter, adj)
    res = np.concatenate([a["x"].T, a["v"].T, a["C"].reshape(n, 9).T, a["F"].reshape(n, 9).T, a["Jp"][None]])
    return res, mb, lb, _clear(mats[0], p.eps, inter["S"], st["Jp"], mu, lam)


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream or None)


def _recorded(d, kind):
    """A runtime at the strained state, its records of d.n_substeps and the adjoint's workspace."""
    from genesis_b200.engine.runtime import runtime_from_descs

    rt = runtime_from_descs([d], sort_interval=0, use_graphs=False)
    F, Cm, jp = _state(d, kind)
    f32 = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float32, device=rt.device)
    n = d.n_particles
    rt.set_state(pos=f32(d.pos), vel=f32(d.vel), C_=f32(Cm.reshape(n, 9)), F=f32(F.reshape(n, 9)), Jp=f32(jp))
    mu, lam = _lame(d)
    rt.set_lame(f32(mu), f32(lam))
    rt.sort()
    m = d.n_substeps

    def size(name):
        b = C.c_uint64()
        nat.check(name, getattr(rt.lib, name)(C.byref(rt.prob), C.byref(b)))
        return b.value

    rs = torch.empty((m,) + tuple(rt.state.shape), dtype=torch.float32, device=rt.device)
    rg = torch.empty(m * size("mpm_record_grid_bytes"), dtype=torch.uint8, device=rt.device)
    ws = torch.empty(size("mpm_adjoint_workspace_bytes"), dtype=torch.uint8, device=rt.device)
    nat.check("mpm_substeps_record", rt.lib.mpm_substeps_record(
        C.byref(rt.prob), C.byref(rt.tables), C.byref(rt.par), rt._ws, m, C.c_void_p(rs.data_ptr()),
        C.c_void_p(rg.data_ptr()), _stream()))
    return rt, rs, rg, ws


def _gpu_adjoint(rt, rs, rg, ws, first, count, adj, lb):
    nat.check("mpm_substeps_adjoint_recorded", rt.lib.mpm_substeps_adjoint_recorded(
        C.byref(rt.prob), C.byref(rt.tables), C.byref(rt.par), first, count, C.c_void_p(rs.data_ptr()),
        C.c_void_p(rg.data_ptr()), C.c_void_p(adj.data_ptr()), C.c_void_p(lb.data_ptr()), C.c_void_p(ws.data_ptr()),
        _stream()))


@pytest.mark.gpu
@pytest.mark.parametrize("kind,kw", MATERIALS, ids=lambda x: str(x)[:30])
def test_each_recorded_substep_matches_the_float64_adjoint(kind, kw):
    from oracle import bridge

    d = _desc(kind, kw, 10, 5)
    rt, rs, rg, ws = _recorded(d, kind)
    n = rt.n
    p, mats, _ = bridge.from_desc(d, np.float64, model_dtype=np.float32)
    mu, lam = rt.mu_p[:n].cpu().numpy(), rt.lam_p[:n].cpu().numpy()
    adj = torch.zeros_like(rt.state)
    adj[:, :n] = torch.as_tensor(_seed_adjoint(n), dtype=torch.float32, device=rt.device)
    worst = {}
    for j in range(d.n_substeps - 1, -1, -1):
        given = adj[:, :n].cpu().numpy().astype(np.float64)
        lb = torch.zeros((3, rt.stride), dtype=torch.float32, device=rt.device)
        _gpu_adjoint(rt, rs, rg, ws, j, 1, adj, lb)
        want, mb, lbo, clear = _oracle_adjoint(p, mats, *_oracle_state(rs[j][:, :n].cpu(), mu, lam), given)
        assert clear.mean() > 0.95
        got = adj[:, :n].cpu().numpy().astype(np.float64)
        pairs = {k: (got[sl], want[sl]) for k, sl in GROUPS.items()}
        pairs.update(mu=(lb[0, :n].cpu().numpy()[None], mb[None]), lam=(lb[1, :n].cpu().numpy()[None], lbo[None]))
        for k, (a, b) in pairs.items():
            use = slice(None) if k in ("x", "v") else clear
            err = np.linalg.norm(a[:, use] - b[:, use]) / max(np.linalg.norm(b[:, use]), 1e-30)
            worst[k] = max(worst.get(k, 0.0), err)
    print(f"\n[recorded adjoint] {kind}: " + ", ".join(f"{k} {v:.1e}" for k, v in worst.items()))
    assert rt.status() == 0
    for k, v in worst.items():
        assert v <= TOL[k], (k, v)


@pytest.mark.gpu
@pytest.mark.parametrize("side", [3, 10, 22])
def test_the_overlapped_chain_equals_its_substeps_one_by_one(side):
    """The three kernels of a substep, and those of the next, overlap in one call: the same records
    taken a substep at a time, each waited for, give the same adjoint but for the order of the
    grid's float sums (roundings of 1e-7 a substep, 24 substeps; 2e-5 is allowed)."""
    kind, kw = MATERIALS[4]
    d = _desc(kind, kw, side, 24)
    rt, rs, rg, ws = _recorded(d, kind)
    n = rt.n
    res = []
    for cuts in ([(0, 24)], [(9, 15), (0, 9)], [(j, 1) for j in range(23, -1, -1)]):
        adj = torch.zeros_like(rt.state)
        adj[:, :n] = torch.as_tensor(_seed_adjoint(n), dtype=torch.float32, device=rt.device)
        lb = torch.zeros((3, rt.stride), dtype=torch.float32, device=rt.device)
        for first, count in cuts:
            _gpu_adjoint(rt, rs, rg, ws, first, count, adj, lb)
            if count == 1:
                torch.cuda.synchronize()
        res.append(torch.cat([adj[:, :n], lb[:2, :n]]).double())
    for r in res[:2]:
        for k, sl in dict(GROUPS, mu=slice(25, 26), lam=slice(26, 27)).items():
            a, b = r[sl], res[2][sl]
            assert float((a - b).norm()) <= 2e-5 * max(float(b.norm()), 1e-30), k
