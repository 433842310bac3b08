"""Runs of substeps with the grid op folded into the particle kernel (rotating grids) against the
separate kernels and the float64 oracle: run lengths around the three-grid rotation, re-sorts inside
a run, runs split at odd places, several environments, one particle, particles that leave their
tile, and a grid left clean for whatever runs next."""

import numpy as np
import pytest
import torch

from genesis_b200 import _native as nat
from genesis_b200 import workloads as W
from genesis_b200.engine import runtime as R

# float32 sums in another order, grown over up to 60 substeps (as in the parity tests)
POS_TOL, VEL_TOL = 1e-6, 1e-4


def _desc(n_side, seed=5, speed=0.5):
    d = W.elastic_cube(n_side=n_side, seed=seed)
    d.vel = np.random.default_rng(seed).normal(0.0, speed, size=d.vel.shape)
    return d


def _runtime(descs, rotate, **kw):
    rt = R.runtime_from_descs(descs, **kw)
    assert rt.prob.flags & nat.PROBF_ROTATE
    if not rotate:
        rt.prob.flags &= ~nat.PROBF_ROTATE
    return rt


def _compare(a, b):
    sa, sb = a.get_state(), b.get_state()
    assert float((sa["pos"] - sb["pos"]).abs().max()) <= POS_TOL
    assert float((sa["vel"] - sb["vel"]).abs().max()) <= VEL_TOL
    assert float((sa["F"] - sb["F"]).abs().max()) <= 1e-5
    assert a.status() == b.status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("runs,interval", [((1,), 50), ((2,), 50), ((3,), 50), ((4, 1, 2, 7), 50), ((60,), 25),
                                           ((20, 13), 8), ((5, 5), 0), ((10,) * 12, 50), ((6, 6, 6, 6, 6), 8)])
@pytest.mark.parametrize("graphs", [False, True])
def test_runs_match_the_separate_kernels(runs, interval, graphs):
    rts = [_runtime([_desc(9), _desc(12, seed=6)], rot, sort_interval=interval, use_graphs=graphs)
           for rot in (True, False)]
    for n in runs:
        for rt in rts:
            rt.substeps(n)
    _compare(*rts)
    mm, _ = rts[0].grid_views()
    assert float(mm.abs().max()) == 0.0  # the grids are clean: the separate kernels can go on from here
    for rt in rts:
        rt.ensure_sorted()
        rt.p2g(), rt.grid_op(), rt.g2p()
        rt._count += 1
        rt.substeps(3)
    _compare(*rts)


@pytest.mark.gpu
@pytest.mark.parametrize("n_side", [1, 3, 20])
def test_matches_oracle(n_side):
    from oracle import bridge, cref

    d = _desc(n_side)
    rt = _runtime([d], True, sort_interval=16)
    rt.substeps(40)
    ref, rc = cref.substeps(*bridge.from_desc(d, np.float64), 40)
    assert rc == 0 and rt.status() == 0
    assert np.abs(rt.get_state(("pos",))["pos"].cpu().numpy() - ref["x"]).max() <= 1e-5


@pytest.mark.gpu
def test_particles_outside_their_tiles():
    rts = []
    for rot in (True, False):
        rt = _runtime([_desc(10, speed=0.0)], rot, sort_interval=0)
        rt.substeps(2)  # binned here, never again
        st = rt.get_state()
        vel = torch.zeros_like(st["vel"])
        vel[::3, 0] = 40.0  # 40 m/s x 1e-4 s: more than a tile's margin within ten substeps
        rt.set_state(vel=vel)
        rt.substeps(12)
        rts.append(rt)
    assert rts[0].fallback_count() > 0
    # fast particles: positions to 1e-6 of the 1 m domain, velocities relative to 40 m/s
    sa, sb = rts[0].get_state(), rts[1].get_state()
    assert float((sa["pos"] - sb["pos"]).abs().max()) <= 1e-5
    assert float((sa["vel"] - sb["vel"]).abs().max()) <= 40 * VEL_TOL


@pytest.mark.gpu
def test_allocation_free_entry_takes_a_flagged_problem():
    import ctypes as C

    d = _desc(10)
    a, b = _runtime([d], True), _runtime([d], False)
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream or None)
    assert a.lib.mpm_substeps_noalloc(C.byref(a.prob), C.byref(a.tables), C.byref(a.par), 7, 5, 0, s) == 0
    b.sort_interval = 5
    b.substeps(7)
    _compare(a, b)


@pytest.mark.gpu
def test_graphs_are_released_while_another_stream_captures():
    rt = _runtime([_desc(8)], True, sort_interval=20)
    for _ in range(5):
        rt.substeps(10)  # captured from the second time on
    torch.cuda.synchronize()
    assert rt._graphs
    x = torch.zeros(4, device="cuda")
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):  # (a scene collected inside somebody's capture)
        x += 1
        rt._drop_graphs()
        x += 1
    g.replay()
    torch.cuda.synchronize()
    assert float(x[0]) == 2.0 and not rt._graphs
    rt.substeps(10)
    assert rt.status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("n_side", [8, 44])  # with the rotating grids, and enough particles for neither
def test_short_runs_can_be_captured_by_the_caller(n_side):
    rts = [R.runtime_from_descs([_desc(n_side)], sort_interval=50) for _ in range(2)]
    for rt in rts:
        for _ in range(5):
            rt.substeps(10)  # phases 0, 10, .. 40
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            rts[0].substeps(10)
        g.replay()
    torch.cuda.current_stream().wait_stream(s)
    rts[1].substeps(10)
    torch.cuda.synchronize()
    _compare(*rts)


@pytest.mark.gpu
def test_profile_times_the_schedule_that_runs():
    for rot in (True, False):
        a, b = (_runtime([_desc(9)], rot, sort_interval=8) for _ in range(2))
        prof = {k: n for k, (ms, n) in a.profile_substeps(20).items()}
        b.substeps(20)
        _compare(a, b)
        # 8 + 8 + 4 substeps, each run from its sort; the grid op by itself only at a run's end
        # where it is folded into the fused kernel
        assert prof == {"sort": 3 * 4, "p2g": 3, "g2p": 3, "g2p2g": 7 + 7 + 3, "grid_op": 3 if rot else 20}
        a.substeps(12)  # and the grids are left clean
        b.substeps(12)
        _compare(a, b)


@pytest.mark.gpu
def test_retune_takes_the_folded_kernel_on_and_off(monkeypatch):
    a = R.runtime_from_descs([_desc(9), _desc(12, seed=6)], sort_interval=16, chunk_particles=256)
    b = _runtime([_desc(9), _desc(12, seed=6)], False, sort_interval=16)
    assert not a.prob.flags & nat.PROBF_ROTATE
    plain = a.workspace_bytes
    for P, rot in ((256, False), (128, True), (256, False), (128, True)):
        a.retune(chunk_particles=P)
        assert bool(a.prob.flags & nat.PROBF_ROTATE) == rot
        assert a.workspace.numel() >= a.workspace_bytes
        assert rot or a.workspace.numel() == plain  # the extra grids are given back
        for rt in (a, b):
            rt.substeps(11)
            rt.substeps(6)
        _compare(a, b)
    monkeypatch.setattr(R, "ROTATE_MAX_PARTICLES", 2000)  # 2,457 particles: too many
    a.retune(chunk_particles=256)
    a.retune(chunk_particles=128)
    assert not a.prob.flags & nat.PROBF_ROTATE


@pytest.mark.gpu
@pytest.mark.parametrize("rotate", [True, False])
def test_short_runs_pay_for_their_graphs(rotate):
    """200 runs of 7 substeps meet a sort interval of 50 at dozens of phases; a loop of 10 meets it at five."""
    a, b = _runtime([_desc(8)], rotate, sort_interval=50), _runtime([_desc(8)], rotate, sort_interval=50)
    b.use_graphs = False
    runs = 0
    for _ in range(200):
        runs += 1 if a._count % 50 + 7 <= 50 else 2
        for rt in (a, b):
            rt.substeps(7)
        if rotate:
            assert len(a._graphs) <= 1 + runs / 16
        else:
            assert len(a._graphs) <= 1 + a._count / 128
    assert len(a._graphs) >= 5
    _compare(a, b)
    c = _runtime([_desc(8)], rotate, sort_interval=50)
    for _ in range(120):
        c.substeps(10)
    assert len(c._graphs) == 5
