"""Accuracy of the kernels' 3x3 SVD on ill-conditioned and nearly degenerate F_tmp.

The SVD is not exposed by itself; two materials read it back after one p2g (particles
isolated, one per 4^3 block, C = 0, so F_tmp = F exactly):

* an ElastoPlastic clamp wider than every singular value (yield_lower = 1, yield_higher =
  1e6: S_new = S) makes p2g write F_new = U S V^T, the kernel's reconstruction of F_tmp.  Its
  error is read in the float64 SVD basis of F: E = U64^T (F_new - F) V64, so E_ii is the error
  of singular value i and E_ij / s_j (i != j) the leak of direction j into i.  F_new is stored
  in float32, so its entries carry rounding of ~6e-8 of the largest singular value s_0: the
  reconstruction is held to 3e-6 s_0, each E_ii to 1e-5 s_i + 2^-20 s_0 and each leak |E_ij|
  to 1e-4 s_j + 2^-20 s_0.
* Snow with its lower clamp at 0.5 (yield_lower = 0.5) writes Jp_new = Jp prod_i s_i / 0.5
  over the singular values below 0.5 (snow.py:62-70): the small singular values' relative
  error, in float32 relative precision.  Held per clamped singular value to 1e-5 relative or
  2^-22 s_0 / s_i, whichever is larger: a float32 SVD of A cannot resolve s_i better than a few
  ulps of s_0 (forming A V alone rounds at that level), and that floor is 2.4e-4 relative at
  s_i = 1e-3 s_0 (measured: 2e-5).

Cases: singular values (1, 1e-2, 1e-3), (1, 1, 1e-3), (1.2, 1e-2, 1e-2 (1 + 1e-4)), nearly
repeated (1, 1 + 1e-6, 0.5) and the well-conditioned range of the benchmark scenes
(0.3 - 1.6).  (Without the kernel's one-sided sweep for ill-conditioned F, the eigenvectors of
F^T F formed in float32 leave the smallest singular value of the 1e-3 case 4e-5 off.)
"""

import numpy as np
import pytest
import torch

from genesis_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _rot(rng, n):
    q = rng.normal(size=(n, 4))
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    w, x, y, z = q.T
    return np.stack([
        np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y)], -1),
        np.stack([2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x)], -1),
        np.stack([2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], -1),
    ], -2)


CASES = {
    "ratio_1e-3": (1.0, 1e-2, 1e-3),
    "two_equal_one_small": (1.0, 1.0, 1e-3),
    "small_pair": (1.2, 1e-2, 1e-2 * (1 + 1e-4)),
    "nearly_repeated": (1.0, 1.0 + 1e-6, 0.5),
}


def _run(F, material=("elastoplastic", dict(use_von_mises=False, yield_lower=1.0, yield_higher=1e6)), key="F"):
    from genesis_b200.engine.runtime import runtime_from_descs

    n = F.shape[0]
    density = 96
    dx = 1.0 / density
    ks = np.stack(np.meshgrid(*[np.arange(1, 16)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    pos = (6 * ks + 1.5) * dx
    d = W.SceneDesc(name="svd", grid_density=density, particle_size=0.01, dt=1e-4, n_substeps=1, pos=pos,
                    vel=np.zeros((n, 3)), mat_idx=np.zeros(n, dtype=np.int64), materials=[material],
                    gravity=(0.0, 0.0, 0.0))
    rt = runtime_from_descs([d], use_graphs=False)
    rt.set_state(pos=pos, C_=np.zeros((n, 3, 3)), F=F)
    rt.sort()
    rt.p2g()
    st = rt.get_state((key,))
    torch.cuda.synchronize()
    return st[key].cpu().numpy().astype(np.float64)


def test_svd_reconstruction_on_ill_conditioned_F():
    rng = np.random.default_rng(17)
    m = 64
    names, Fs, sig = [], [], []
    for name, s in CASES.items():
        S = np.tile(np.asarray(s), (m, 1))
        names += [name] * m
        sig.append(S)
    S = rng.uniform(0.3, 1.6, size=(m, 3))
    names += ["benchmark_range"] * m
    sig.append(S)
    sig = np.concatenate(sig)
    n = sig.shape[0]
    U0, V0 = _rot(rng, n), _rot(rng, n)
    F = U0 @ (sig[:, :, None] * np.swapaxes(V0, 1, 2))
    F32 = F.astype(np.float32).astype(np.float64)  # what the kernel is given
    Fn = _run(F32)
    U, s, Vt = np.linalg.svd(F32)
    E = np.swapaxes(U, 1, 2) @ (Fn - F32) @ np.swapaxes(Vt, 1, 2)
    # Snow clamped below 0.5: Jp_new = prod over s_i < 0.5 of s_i / 0.5 (Jp = 1)
    Jp = _run(F32, ("snow", dict(yield_lower=0.5, yield_higher=1e6)), key="Jp")
    low = s < 0.5
    want = np.prod(np.where(low, s / 0.5, 1.0), axis=1)
    names = np.array(names)
    idx = np.arange(3)
    for name in list(CASES) + ["benchmark_range"]:
        sel = names == name
        s0 = s[sel, 0][:, None]
        rec = np.abs(Fn[sel] - F32[sel]).max() / s[sel, 0].max()
        dE = np.abs(np.diagonal(E[sel], axis1=1, axis2=2))
        ok_s = dE <= 1e-5 * s[sel] + 2.0**-20 * s0
        leak = np.abs(E[sel]) / (1e-4 * s[sel][:, None, :] + 2.0**-20 * s0[:, :, None])  # <= 1 passes
        leak[:, idx, idx] = 0
        n_low = low[sel].sum(1)
        jrel = np.abs(Jp[sel] - want[sel]) / want[sel]
        print(f"\n[svd] {name}: max|U S V^T - F| / s0 = {rec:.2e}; per-singular-value |E_ii| / s_i "
              f"{(dE / s[sel]).max(0)}; worst leak / (1e-4 s + 2^-20 s0) = {leak.max():.2e}; Snow Jp_new rel. err "
              f"{jrel.max():.2e} over {int(n_low.max())} clamped singular values")
        assert rec < 3e-6, (name, rec)
        assert ok_s.all(), (name, (dE / s[sel]).max(0))
        assert leak.max() <= 1.0, (name, leak.max())
        # each clamped s_i's relative error: 1e-5, or float32's own floor for it, a few ulps of
        # s_0 over s_i (forming B = A V in float32 already costs that), whichever is larger
        bound = np.where(low[sel], np.maximum(1e-5, 2.0**-22 * s0 / s[sel]), 0.0).sum(1)
        assert (jrel <= np.maximum(bound, 1e-6)).all(), (name, jrel.max(), bound.max())


def _stretched(rng, sig):
    n = len(sig)
    F = _rot(rng, n) @ (sig[:, :, None] * np.swapaxes(_rot(rng, n), 1, 2))
    return F.astype(np.float32).astype(np.float64)


@pytest.mark.parametrize("ratio", [1.4, 2.0, 3.9])
def test_moderate_stretches_lose_nothing_off_the_diagonal(ratio):
    """U S V^T of stretches of up to 4 : 1 in the float64 basis: the entries off the diagonal are the
    large columns' remainders in the small ones' directions, a rounding (6e-8) or so of s_0 where the
    large columns are orthogonalised first, the ratio times that where a small one is.  Root mean
    square over 3,375 particles within 1e-7."""
    rng = np.random.default_rng(3)
    n = 3375
    t = rng.uniform(0.0, 1.0, size=(n, 3))
    t[:, 0], t[:, 1] = 0.0, 1.0
    sig = np.take_along_axis(1.1 * ratio ** (t - 0.5), np.argsort(rng.random((n, 3)), 1), 1)
    F = _stretched(rng, sig)
    U, s, Vt = np.linalg.svd(F)
    E = np.swapaxes(U, 1, 2) @ (_run(F) - F) @ np.swapaxes(Vt, 1, 2)
    E[:, [0, 1, 2], [0, 1, 2]] = 0.0
    rms = np.sqrt((E ** 2).mean())
    print(f"\n[svd] ratio {ratio}: rms off the diagonal {rms:.2e}")
    assert rms <= 1e-7


@pytest.mark.parametrize("sig", [(1.0, 1.0, 1e-2), (1.3, 0.9, 0.2), (2.8, 1.0, 1.0)])
def test_liquid_volume_of_stretched_particles(sig):
    """An inviscid Liquid takes J = det F_tmp alone, with no rotation to separate the columns, and writes
    F_new = J^(1/3) I.  Its relative error: a rounding (6e-8) of s_0 in the smallest singular value and
    a few in the others; three times 6e-8 s_0 / s_2 + 1e-6 is allowed."""
    rng = np.random.default_rng(8)
    F = _stretched(rng, np.tile(np.array(sig), (3375, 1)))
    Fn = _run(F, ("liquid", dict(E=1e5, nu=0.2)))
    err = np.abs(Fn[:, 0, 0] ** 3 / np.linalg.det(F) - 1.0).max()
    print(f"\n[svd] liquid {sig}: J rel. err {err:.2e}")
    assert err <= 3 * 6e-8 * max(sig) / min(sig) + 1e-6
