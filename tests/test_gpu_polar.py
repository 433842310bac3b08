"""Elastic and Liquid particles on both sides of the conditions under which a warp takes J and the polar
rotation of F_tmp without an SVD: det F_tmp > 1e-6, |F_tmp|_F^6 < 108 det^2 (singular values (a, 1, 1)
pass for a in [0.29, 2.68]).

Alone: one substep of strained particles at rest (C = 0, so F_tmp = F) against the float64 oracle; every
particle has its own stretch of the grid, so its C shows its own stress.  Tolerance 3e-5 of the
particle's largest |C|, taken as at least a hundredth of the scene's (an unstrained particle's is
rounding), for v of |v| + dx |C|: the rotation's rounding of 1e-7 against ordinary strains of 5e-2 (2e-6
of the stress), up to 1e-6 where the stretch is 3.4 : 1 or the determinant is small, and the scatter's
fixed-point sums (5e-7 of the bound a node, 27 nodes).  (J of a Liquid by itself: test_gpu_svd.py.)

One lane of a full warp: the particle among 31 ordinary ones (refused, it sends its whole warp to the
SVD), and also with a Snow particle beside it (which needs the SVD anyway).  There v and C are
quotients of sums that cancel, and the scatter's rounding shows in them at 1e-4 whichever way the
stress was computed; compared instead is the first moment of the group's momentum about its middle,
which is sum_p A_p dx^2 / 4 (A the affine momentum, here the scaled stress): a sum of the lanes'
stresses.  Its rounding: each of 32 x 27 contributions to half a quantum q of the fixed-point
sums, q <= 256 B / 2^29 with B = 1.5 dx max sum_j |A_ij| the bound on a contribution, about 2 dx from the
middle: 8e-6 B dx for independent roundings, five times that is allowed; a lane's own stress is some
0.05 B dx."""

import numpy as np
import pytest
import torch

from genesis_b200 import workloads as W

STRETCHES = [
    (0.28, 1, 1), (0.2885, 1, 1), (0.2905, 1, 1), (0.30, 1, 1),
    (2.60, 1, 1), (2.675, 1, 1), (2.688, 1, 1), (2.80, 1, 1),
    (1, 1, 1e-2), (1, 1e-2, 1e-2), (9.8e-3, 9.8e-3, 9.8e-3), (1.03e-2, 1.03e-2, 1.03e-2),
    (1, 1, 1), (1.3, 1.0, 0.8),
]
INVERTED = [(1, 0.9, -1e-3), (1.1, 0.9, -0.2), (0.02, 0.015, -0.01)]  # det slightly and clearly negative
MATERIALS = [
    ("elastic", dict(E=1e5, nu=0.3)),
    ("elastic", dict(E=1e5, nu=0.3, model="neohooken")),
    ("liquid", dict(E=1e5, nu=0.2)),
    ("liquid", dict(E=1e5, nu=0.2, viscous=True)),
]
IDS = ["corotated", "neohooken", "liquid", "viscous"]
DENSITY, REPEATS = 96, 6
CORNERS = [(i, j, k) for i in range(1, 11) for j in range(1, 11) for k in range(1, 11)]  # groups of 8^3 nodes


def _rotation(rng):
    q, r = np.linalg.qr(rng.normal(size=(3, 3)))
    q = q * np.sign(np.diag(r))
    return q if np.linalg.det(q) > 0 else -q


def _scene(kind, kw, layout, seed=21):
    """(desc, F, group of each particle)"""
    rng = np.random.default_rng(seed)
    # an inverted Liquid's or neo-Hookean's F and stress are NaN by the model
    stretches = STRETCHES + (INVERTED if kind == "elastic" and kw.get("model") != "neohooken" else [])
    pos, F, mat, group = [], [], [], []
    for g, s in enumerate(stretches * REPEATS):
        others = {"alone": 0, "among": 31, "beside_snow": 31}[layout]
        for q in range(others + 1):
            pos.append((8 * np.array(CORNERS[g]) + 0.5 + rng.uniform(0.4, 3.6, size=3)) / DENSITY)
            if q == others // 2:
                F.append(_rotation(rng) @ np.diag(s).astype(float) @ _rotation(rng).T)
            else:
                F.append(np.eye(3) + 0.05 * rng.normal(size=(3, 3)))
            mat.append(1 if layout == "beside_snow" and q == 0 else 0)
            group.append(g)
    d = W.SceneDesc(name="polar", grid_density=DENSITY, particle_size=0.5 / DENSITY, dt=1e-4, n_substeps=1,
                    pos=np.array(pos, dtype=np.float32).astype(np.float64), vel=np.zeros((len(pos), 3)),
                    mat_idx=np.array(mat), materials=[(kind, dict(kw)), ("snow", dict(E=1e5))])
    return d, np.array(F, dtype=np.float32).astype(np.float64), np.array(group)


@pytest.mark.gpu
@pytest.mark.parametrize("kind,kw", MATERIALS, ids=IDS)
def test_stress_on_both_sides_of_each_condition(kind, kw):
    from genesis_b200.engine.runtime import runtime_from_descs
    from oracle import bridge, cref

    d, F, group = _scene(kind, kw, "alone")
    rt = runtime_from_descs([d])
    rt.set_state(F=torch.as_tensor(F, dtype=torch.float32, device=rt.device))
    rt.substeps(1)
    got = {k: v.cpu().numpy().astype(np.float64) for k, v in rt.get_state(("vel", "C")).items()}
    assert rt.status() == 0
    p, mats, st = bridge.from_desc(d, np.float64, model_dtype=np.float32)
    st["F"] = F.copy()
    ref, rc = cref.substeps(p, mats, st, 1)
    assert rc == 0
    n = group.max() + 1
    worst = lambda a: np.array([np.abs(a[group == g]).max() for g in range(n)])
    C, Cr = got["C"].reshape(-1, 3, 3), ref["C"]
    sC = np.maximum(worst(Cr), 1e-2 * np.abs(Cr).max())
    eC = worst(C - Cr) / sC
    eV = worst(got["vel"] - ref["v"]) / (worst(ref["v"]) + sC / DENSITY)
    print(f"\n[polar] {kind}: C {eC.max():.1e} (group {eC.argmax()}), v {eV.max():.1e}")
    assert eC.max() <= 3e-5 and eV.max() <= 3e-5


@pytest.mark.gpu
@pytest.mark.parametrize("layout", ["among", "beside_snow"])
@pytest.mark.parametrize("kind,kw", MATERIALS, ids=IDS)
def test_one_lane_of_a_full_warp(kind, kw, layout):
    from genesis_b200.engine.runtime import block_major_to_dense, runtime_from_descs
    from oracle import bridge
    from oracle import mpm_adjoint as A

    d, F, group = _scene(kind, kw, layout)
    rt = runtime_from_descs([d])
    rt.set_state(F=torch.as_tensor(F, dtype=torch.float32, device=rt.device))
    rt.sort()
    rt.p2g()
    mm = block_major_to_dense(rt.grid_views()[0].cpu().numpy().astype(np.float64), rt.specs[0], 0)
    assert rt.status() == 0
    p, mats, st = bridge.from_desc(d, np.float64, model_dtype=np.float32)
    st["F"] = F.copy()
    lame = lambda name: np.array([getattr(mats[m], name) for m in d.mat_idx])
    _, inter = A.forward_materials(p, mats, st, lame("mu"), lame("lam"))
    Ap, dx = inter["A"], p.dx
    at = (np.stack(np.meshgrid(*[np.arange(8)] * 3, indexing="ij"), -1).reshape(-1, 3) - 2.5) * dx
    worst = 0.0
    for g in range(group.max() + 1):
        c = 8 * np.array(CORNERS[g])
        mom = mm[c[0]:c[0] + 8, c[1]:c[1] + 8, c[2]:c[2] + 8, :3].reshape(-1, 3)
        lanes = Ap[group == g]
        B = 1.5 * dx * np.abs(lanes).sum(2).max()
        worst = max(worst, np.abs(mom.T @ at - lanes.sum(0) * dx * dx / 4).max() / (B * dx))
    print(f"\n[polar] {kind} {layout}: moment {worst:.1e} B dx")
    assert worst <= 4e-5
