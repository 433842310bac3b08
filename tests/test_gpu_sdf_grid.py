"""The signed-distance grid kernels on meshes and grids where they could go wrong: sizes that leave
bricks partly outside, fewer and more faces than one shared-memory stage holds, open meshes
(fractional winding numbers), nodes far outside, grids away from the origin with different steps per
axis, invalid faces.  Grids below 75,000 nodes take a warp per node (the first cases), larger ones
bricks of nodes (the later ones, where the brick's bounds on distance and winding number, its faces
near and far and its fallback to every face decide).  Against the float64 oracle: distances to 4e-6
of the coordinates' magnitude (a few float32 roundings of a point-triangle distance), the side
wherever the winding number is not within 1e-3 of 1/2."""

import ctypes as C

import numpy as np
import pytest
import torch

from genesis_b200 import _native as nat
from oracle import sdf_ref


def _sphere(nu, nv, open_below=None):
    th, al = np.pi * np.arange(1, nv) / nv, 2 * np.pi * np.arange(nu) / nu
    T, A = np.meshgrid(th, al, indexing="ij")
    v = np.stack([0.4 * np.sin(T) * np.cos(A), 0.3 * np.sin(T) * np.sin(A), 0.5 * np.cos(T)], -1).reshape(-1, 3)
    v = np.concatenate([v, [[0, 0, 0.5], [0, 0, -0.5]]])
    f = []
    for j in range(nu):
        m = (j + 1) % nu
        f += [(len(v) - 2, j, m), (len(v) - 1, (nv - 2) * nu + m, (nv - 2) * nu + j)]
        for i in range(nv - 2):
            a, b, c, d = i * nu + j, i * nu + m, (i + 1) * nu + j, (i + 1) * nu + m
            f += [(a, c, b), (b, c, d)]
    f = np.array(f, dtype=np.int32)
    if open_below is not None:
        f = f[v[f].mean(1)[:, 2] > open_below]
    return v, f


def _grid(v, f, origin, step, res):
    lib = nat.load()
    vt = torch.as_tensor(v.astype(np.float32), device="cuda")
    ft = torch.as_tensor(f, device="cuda")
    out = torch.empty(tuple(res), dtype=torch.float32, device="cuda")
    rc = lib.mpm_sdf_grid(C.c_void_p(vt.data_ptr()), len(v), C.c_void_p(ft.data_ptr()), len(f),
                          (C.c_float * 3)(*origin), (C.c_float * 3)(*step), (C.c_int32 * 3)(*res),
                          C.c_void_p(out.data_ptr()), C.c_void_p(torch.cuda.current_stream().cuda_stream or None))
    assert rc == 0
    return out.cpu().numpy().astype(np.float64)


@pytest.mark.gpu
@pytest.mark.parametrize("nu,nv,open_below,origin,step,res", [
    (5, 3, None, (-0.6, -0.6, -0.6), (0.1, 0.1, 0.1), (13, 13, 13)),
    (24, 9, None, (-0.6, -0.6, -0.6), (0.05, 0.06, 0.07), (25, 19, 17)),
    (40, 17, None, (-2.0, -0.2, -0.7), (0.3, 0.02, 0.045), (9, 21, 33)),
    (24, 9, 0.1, (-0.6, -0.6, -0.6), (0.05, 0.05, 0.05), (25, 25, 25)),
    (16, 8, -0.3, (-0.5, -0.4, -0.8), (0.08, 0.0, 0.08), (12, 1, 20)),
])
def test_grid_matches_oracle(nu, nv, open_below, origin, step, res):
    v, f = _sphere(nu, nv, open_below)
    v = v.astype(np.float32).astype(np.float64)
    got = _grid(v, f, origin, step, res)
    o, s = np.float32(origin), np.float32(step)
    ax = [(o[d] + s[d] * np.arange(res[d], dtype=np.float32)).astype(np.float64) for d in range(3)]
    p = np.stack(np.meshgrid(*ax, indexing="ij"), -1).reshape(-1, 3)
    want = sdf_ref.signed_distance(p, v, f).reshape(res)
    scale = max(np.abs(p).max(), 0.5)
    assert np.abs(np.abs(got) - np.abs(want)).max() <= 4e-6 * scale
    w = np.zeros(len(p))
    for t in f:
        w += sdf_ref._solid_angle(p, v[t[0]], v[t[1]], v[t[2]])
    clear = (np.abs(np.abs(w) / (4 * np.pi) - 0.5) > 1e-3).reshape(res) & (np.abs(want) > 4e-6 * scale)
    assert clear.mean() > 0.9
    assert (np.sign(got) == np.sign(want))[clear].all()
    assert (got < 0).any() or open_below is not None


@pytest.mark.gpu
def test_invalid_faces_are_skipped_and_none_left_is_far_outside():
    v, f = _sphere(24, 9)
    bad = np.concatenate([[[0, 1, len(v)]], f, [[-1, 0, 1]]]).astype(np.int32)
    args = ((-0.6,) * 3, (0.11,) * 3, (11, 11, 11))
    assert np.array_equal(_grid(v, bad, *args), _grid(v, f, *args))
    assert (_grid(v, np.full((3, 3), len(v), dtype=np.int32), *args) > 1e18).all()


BRICK_CASES = [
    # closed, 384 faces, no edge a multiple of a brick's
    (24, 9, None, (-0.6, -0.6, -0.7), (0.026, 0.027, 0.033), (47, 45, 43)),
    # 20 large faces: every face near every brick
    (5, 3, None, (-0.5, -0.45, -0.6), (0.0165, 0.026, 0.031), (61, 35, 39)),
    # 1,280 faces, most nodes far outside, steps of 1:15
    (40, 17, None, (-2.0, -0.42, -0.7), (0.09, 0.006, 0.033), (45, 141, 43)),
    # open meshes: the side turns where the winding number passes 1/2, away from any face
    (24, 9, 0.1, (-0.6, -0.6, -0.6), (0.0231, 0.0291, 0.033), (53, 41, 37)),
    (40, 17, -0.3, (-0.5, -0.4, -0.8), (0.02, 0.02, 0.02), (50, 41, 66)),
    # planes and a zero step
    (16, 8, -0.3, (-0.5, -0.4, -0.8), (0.0035, 0.0, 0.005), (290, 1, 270)),
    (16, 8, -0.3, (-0.5, 0.02, -0.8), (0.0035, 0.0, 0.005), (290, 1, 270)),
    (24, 9, None, (0.1, -0.4, -0.55), (0.0, 0.003, 0.004), (2, 151, 257)),
]


@pytest.mark.gpu
@pytest.mark.parametrize("nu,nv,open_below,origin,step,res", BRICK_CASES)
def test_bricks_match_oracle(nu, nv, open_below, origin, step, res):
    """6,000 nodes of each grid: those nearest the surface, those whose winding number is nearest
    1/2, and a random third."""
    assert np.prod(res) >= 75_000
    v, f = _sphere(nu, nv, open_below)
    v = v.astype(np.float32).astype(np.float64)
    got = _grid(v, f, origin, step, res).reshape(-1)
    o, s = np.float32(origin), np.float32(step)
    ax = [(o[d] + s[d] * np.arange(res[d], dtype=np.float32)).astype(np.float64) for d in range(3)]
    p = np.stack(np.meshgrid(*ax, indexing="ij"), -1).reshape(-1, 3)
    wind = _winding(p, v, f)
    at = np.unique(np.concatenate([np.argsort(np.abs(got))[:2000], np.argsort(np.abs(wind - 0.5))[:2000],
                                   np.random.default_rng(1).choice(len(p), 2000, replace=False)]))
    want = sdf_ref.signed_distance(p[at], v, f)
    scale = max(np.abs(p).max(), 0.5)
    assert np.abs(np.abs(got[at]) - np.abs(want)).max() <= 4e-6 * scale
    # the side of every node
    clear = (np.abs(wind - 0.5) > 1e-3) & (np.abs(got) > 4e-6 * scale)
    assert clear.mean() > 0.9
    assert (np.sign(got) == np.where(wind > 0.5, -1.0, 1.0))[clear].all()
    assert (got > 0).any() and ((got < 0).any() or open_below is not None)


def _winding(p, v, f):
    """|winding number| of the oracle's solid angles at every node, on the GPU in float64 (its numpy
    takes seconds a hundred faces)."""
    P = torch.as_tensor(p, device="cuda")
    w = torch.zeros(len(p), dtype=torch.float64, device="cuda")
    for t in f:
        r = [torch.as_tensor(v[k], device="cuda") - P for k in t]
        n = [q.norm(dim=1) for q in r]
        det = (r[0] * torch.linalg.cross(r[1], r[2])).sum(1)
        den = n[0] * n[1] * n[2] + (r[0] * r[1]).sum(1) * n[2] + (r[0] * r[2]).sum(1) * n[1] + (r[1] * r[2]).sum(1) * n[0]
        w += 2 * torch.atan2(det, den)
    return w.abs().cpu().numpy() / (4 * np.pi)


@pytest.mark.gpu
def test_bricks_skip_invalid_faces():
    v, f = _sphere(24, 9)
    bad = np.concatenate([[[0, 1, len(v)]], f[:200], [[-1, 0, 1], [len(v) + 7, 2, 3]], f[200:]]).astype(np.int32)
    args = ((-0.6, -0.6, -0.6), (0.028, 0.028, 0.028), (43, 44, 42))
    got, want = _grid(v, bad, *args), _grid(v, f, *args)
    assert np.abs(np.abs(got) - np.abs(want)).max() <= 1e-6  # the stages hold other faces: another order of sums
    assert (np.sign(got) == np.sign(want))[np.abs(want) > 1e-5].all()
    assert (_grid(v, np.full((3, 3), len(v), dtype=np.int32), *args) > 1e18).all()
