"""The signed-distance grid kernel on meshes and grids where its brick bounds could go wrong:
sizes that leave bricks partly outside, fewer and more faces than one shared-memory stage holds, an
open mesh (fractional winding numbers), nodes far outside, a grid away from the origin with
different steps per axis.  Against the float64 oracle: distances to 4e-6 of the coordinates'
magnitude (a few float32 roundings of a point-triangle distance), the side wherever the winding
number is not within 1e-3 of 1/2."""

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
