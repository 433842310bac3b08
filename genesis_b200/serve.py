"""Serving: continuous batching of MPM rollout requests on one GPU.

Requests (a scene plus a number of substeps) arrive over time.  The server keeps every
admitted rollout's particle state resident in HBM, admits queued requests as soon as
slots and the memory budget allow, and advances all admitted rollouts together in the
batched kernels (one instance per rollout), a tick of at most ``tick_substeps`` substeps
at a time.  Between ticks finished rollouts are read back and retired, rollouts whose
instance status shows NaN are evicted with an error, newly admitted ones are packed in,
and the particle state of the continuing ones is carried over device to device.
A request's result does not depend on what it shares the GPU with: instances never
share grid memory or work items.  There is no counterpart in the reference.
"""

from __future__ import annotations

import collections
import dataclasses
import math
import time

import numpy as np
import torch

from . import _native as nat
from . import workloads as W
from .engine.runtime import MPMRuntime, rotate_bytes, spec_from_desc
from .materials import MPM


def estimate_bytes(desc, chunk_particles: int = 128) -> int:
    """HBM a request holds while admitted: particle state and ids, plus its share of the
    workspace (grids, bins, chunk table, permutation scratch)."""
    n = desc.n_particles
    res = desc.grid_res
    nblk = (res + nat.MPM_BLOCK - 1) // nat.MPM_BLOCK
    blocks = nblk**3
    per_particle = 25 * 4 + 10 + (8 + 25 * 4 + 14)  # state+ids, sort keys/ranks + permutation scratch
    per_block = nat.MPM_BLOCK**3 * 32 + 24  # two float4 grids + flags/active/bins
    chunks = (n // chunk_particles + min(n, blocks) + 1) * 16
    return int(n * per_particle + blocks * per_block + chunks)


def _upload(a, dtype, dev):
    """Host array -> device tensor through pinned memory, without waiting for the stream
    (a copy from pageable memory would block the host until the GPU reaches it)."""
    h = torch.as_tensor(np.asarray(a)).to(dtype).pin_memory()
    return h.to(dev, non_blocking=True)


def _download(t):
    """Device tensor -> pinned host tensor, enqueued on the current stream."""
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t, non_blocking=True)
    return h


@dataclasses.dataclass
class Result:
    rid: int
    arrival: float
    admitted: float | None = None
    finished: float | None = None
    pos: np.ndarray | None = None
    vel: np.ndarray | None = None
    error: str | None = None

    @property
    def latency(self) -> float | None:
        return None if self.finished is None else self.finished - self.arrival


@dataclasses.dataclass
class _Slot:
    req: W.Request
    remaining: int
    bytes: int
    state: dict | None = None  # device tensors in API order while being repacked
    retired: bool = False  # finished or evicted; a hole until the next repack
    spec: object = None  # InstanceSpec, built once at admission
    mats: list | None = None


class AdmissionQueue:
    """FIFO admission against a byte budget and a slot cap (head-of-line order kept)."""

    def __init__(self, budget_bytes: float, max_active: int, chunk_particles: int = 128):
        self.budget = float(budget_bytes)
        self.max_active = int(max_active)
        self.chunk = chunk_particles
        self.pending: collections.deque = collections.deque()
        self.in_use = 0
        self.peak_in_use = 0

    def push(self, req) -> str | None:
        need = estimate_bytes(req.scene, self.chunk)
        if need > self.budget:
            return f"request needs {need} bytes, more than the whole budget ({int(self.budget)})"
        self.pending.append((req, need))
        return None

    def admissible_particles(self, n_active: int) -> int:
        """Particles of the requests pop_admissible would admit now (nothing is popped)."""
        total, used, k = 0, self.in_use, 0
        for req, need in self.pending:
            if n_active + k >= self.max_active or used + need > self.budget:
                break
            used += need
            k += 1
            total += req.scene.n_particles
        return total

    def pop_admissible(self, n_active: int) -> list:
        out = []
        while self.pending and n_active + len(out) < self.max_active and self.in_use + self.pending[0][1] <= self.budget:
            req, need = self.pending.popleft()
            self.in_use += need
            self.peak_in_use = max(self.peak_in_use, self.in_use)
            out.append((req, need))
        return out

    def release(self, need: int):
        self.in_use -= need


class MPMServer:
    def __init__(self, budget_bytes: float = 150e9, tick_substeps: int = 50, max_active: int = 512,
                 chunk_particles: int = 256, sort_interval: int = 100, keep_results: bool = True,
                 use_graphs: bool = False, admit_wait: float = 0.2, admit_ratio: float = 0.25,
                 min_live_particles: int = 2_000_000):
        """chunk_particles / sort_interval: the launch configuration of every layout; 256-particle
        work items re-sorted every 100 substeps is what the autotuner picks for the 256-scene
        batch, and at saturation on the serving mix it measured 6.58e9 particle-substeps/s
        against 6.14e9 for 128 / 50.  admit_wait > 0 batches admissions: while at least min_live_particles are being
        advanced, queued requests join (which costs a repack of every live rollout) only
        once the particles that fit now reach admit_ratio of the live ones, or once the
        oldest has waited admit_wait seconds and the last repack is admit_wait seconds old.
        admit_wait = 0 admits at every tick.  A tick advances up to tick_substeps substeps,
        split where live rollouts finish (each is read back and retired, stream-ordered, at
        its own last substep), with one wait for the GPU per tick."""
        self.tick = int(tick_substeps)
        self.admit_wait = float(admit_wait)
        self.admit_ratio = float(admit_ratio)
        self.min_live_particles = int(min_live_particles)
        self.queue = AdmissionQueue(budget_bytes, max_active, chunk_particles)
        self.chunk = chunk_particles
        self.sort_interval = sort_interval
        self.keep_results = keep_results
        self.use_graphs = use_graphs  # runtimes are short-lived; capture would not amortise
        self.rt: MPMRuntime | None = None
        self.active: list[_Slot] = []
        self.ticks = 0
        self.repacks = 0
        self.repack_s = 0.0  # host seconds spent building layouts
        self.particle_substeps = 0
        self.substeps_run = 0  # substeps enqueued, over every tick

    # ------------------------------------------------------------------ packing
    def _repack(self, new_slots):
        """Build a runtime for the live rollouts plus new_slots: continuing rollouts keep
        their device state; retired ones (holes) are dropped."""
        t_start = time.perf_counter()
        try:
            self._repack_layout(new_slots)
        finally:
            self.repack_s += time.perf_counter() - t_start

    def _repack_layout(self, new_slots):
        live = [s for s in self.active if not s.retired]
        if self.rt is not None and live:
            exported = self.rt.export_instances()
            for slot, st in zip(self.active, exported):
                if not slot.retired:
                    slot.state = st
        self.rt = None
        self.active = live + list(new_slots)
        if not self.active:
            return
        dev = torch.device("cuda")
        specs = []
        parts = {k: [] for k in ("pos", "vel", "C", "F", "Jp", "active", "mat")}
        for slot in self.active:
            d = slot.req.scene
            if slot.spec is None:
                slot.mats = W.make_materials(d, MPM)
                slot.spec = spec_from_desc(d, slot.mats)
            mats = slot.mats
            specs.append(slot.spec)
            if slot.state is None:  # newly admitted: upload its initial state
                n = d.n_particles
                djp = np.array([m.default_Jp for m in mats], dtype=np.float32)[d.mat_idx]
                slot.state = {
                    "pos": _upload(d.pos, torch.float32, dev),
                    "vel": _upload(d.vel, torch.float32, dev),
                    "C": torch.zeros((n, 9), dtype=torch.float32, device=dev),
                    "F": torch.eye(3, dtype=torch.float32, device=dev).reshape(1, 9).repeat(n, 1),
                    "Jp": _upload(djp, torch.float32, dev),
                    "active": torch.ones(n, dtype=torch.bool, device=dev),
                    "mat": _upload(d.mat_idx, torch.uint8, dev),
                }
            for k in parts:
                v = slot.state[k]
                parts[k].append(v.reshape(v.shape[0], -1) if k in ("C", "F") else v)
        # (128-particle layouts may take two more grids, which the requests' estimates do not hold:
        # where the budget has no room for them the layout does without)
        extra = rotate_bytes(sum(sp.n_blocks for sp in specs))
        self.rt = MPMRuntime(specs, chunk_particles=self.chunk, sort_interval=self.sort_interval,
                             use_graphs=self.use_graphs, rotate=self.queue.in_use + extra <= self.queue.budget)
        self.rt.load_state(torch.cat(parts["pos"]), torch.cat(parts["vel"]), torch.cat(parts["C"]),
                           torch.cat(parts["F"]), torch.cat(parts["Jp"]), torch.cat(parts["active"]),
                           torch.cat(parts["mat"]))
        for slot in self.active:
            slot.state = None
        self.repacks += 1

    def _retire(self, k):
        """Drop rollout k from the work without repacking: its particles go inactive."""
        slot = self.active[k]
        slot.retired = True
        off = self.rt.instance_offsets[k]
        n = slot.req.scene.n_particles
        idx = torch.arange(off, off + n, dtype=torch.int32, device=self.rt.device)
        self.rt.set_particles_active(idx, torch.zeros(n, dtype=torch.uint8, device=self.rt.device))
        self.queue.release(slot.bytes)

    # ------------------------------------------------------------------ loop
    def serve(self, requests, realtime: bool = True, on_result=None) -> list[Result]:
        """Run the request stream to completion.  With realtime=True a request becomes
        visible at its arrival time (seconds after the call starts); with realtime=False
        all requests are visible at t=0 (throughput runs).

        The loop is pipelined: a tick's substeps, the read of its per-instance statuses and
        of the results of the rollouts it completes are enqueued first; retiring those
        rollouts, admitting queued requests and repacking (all stream-ordered after the
        tick) then run on the host while the GPU works, and only then does the host wait
        for the tick.  A rollout whose status shows NaN is evicted from whatever layout it
        is in by then."""
        reqs = sorted(requests, key=lambda r: r.arrival)
        results = {r.rid: Result(r.rid, r.arrival if realtime else 0.0) for r in reqs}
        t0 = time.perf_counter()
        clock = lambda: time.perf_counter() - t0
        bad = nat.MPM_STATUS_NAN | nat.MPM_STATUS_NONFINITE_VEL
        i = 0
        n_live = lambda: sum(1 for s in self.active if not s.retired)
        last_repack = -math.inf

        def push_arrivals():
            nonlocal i
            now = clock()
            while i < len(reqs) and (not realtime or reqs[i].arrival <= now):
                err = self.queue.push(reqs[i])
                if err:
                    results[reqs[i].rid].error = err
                    results[reqs[i].rid].finished = now
                i += 1

        def admit():
            nonlocal last_repack
            if not self.queue.pending:
                return False
            if self.admit_wait > 0.0 and n_live():
                live_p = sum(s.req.scene.n_particles for s in self.active if not s.retired)
                if live_p >= self.min_live_particles:
                    fit_p = self.queue.admissible_particles(n_live())
                    if fit_p == 0:
                        return False
                    oldest = self.queue.pending[0][0]
                    waited = clock() - (oldest.arrival if realtime else 0.0)
                    stale = waited >= self.admit_wait and clock() - last_repack >= self.admit_wait
                    if fit_p < self.admit_ratio * live_p and not stale:
                        return False
            admitted = self.queue.pop_admissible(n_live())
            if not admitted:
                return False
            last_repack = clock()
            now = clock()
            new_slots = []
            for req, need in admitted:
                results[req.rid].admitted = now
                new_slots.append(_Slot(req, int(req.scene.n_substeps), need))
            self._repack(new_slots)
            return True

        while i < len(reqs) or self.queue.pending or n_live():
            push_arrivals()
            if not n_live() and not admit():
                self.rt = None
                self.active = []
                if i < len(reqs) and realtime:
                    time.sleep(max(0.0, min(0.05, reqs[i].arrival - clock())))
                continue
            # ---- enqueue one tick (segments ending where live rollouts finish, each finished
            # rollout read back and retired right after its last substep), then the read of
            # the instances' statuses
            tick_slots = [s for s in self.active if not s.retired]
            tick_index = {id(s): k for k, s in enumerate(self.active)}
            T = min(self.tick, max(s.remaining for s in tick_slots))
            fin_host = {}
            done = 0
            while True:
                finishing = [s for s in tick_slots if s.remaining == 0 and not s.retired]
                if finishing and self.keep_results:
                    st = self.rt.get_state(("pos", "vel"))
                    offs = self.rt.instance_offsets
                    for s in finishing:
                        k = tick_index[id(s)]
                        sl = slice(offs[k], offs[k] + s.req.scene.n_particles)
                        fin_host[id(s)] = tuple(_download(st[key][sl]) for key in ("pos", "vel"))
                for s in finishing:
                    self._retire(tick_index[id(s)])
                running = [s for s in tick_slots if s.remaining > 0]
                if not running or done >= T:
                    break
                seg = min(T - done, min(s.remaining for s in running))
                self.rt.substeps(seg)
                self.particle_substeps += seg * sum(s.req.scene.n_particles for s in running)
                self.substeps_run += seg
                done += seg
                for s in running:
                    s.remaining -= seg
            self.ticks += 1
            status_host, status_ev = self.rt.instance_status_enqueue(clear=True)
            # ---- host work while the tick runs (all GPU work it issues is stream-ordered)
            push_arrivals()
            admit()
            # ---- wait for the tick
            status_ev.synchronize()
            status = status_host.numpy().view(np.uint32)
            now = clock()
            for s in tick_slots:
                if not status[tick_index[id(s)]] & bad and s.remaining:
                    continue
                r = results[s.req.rid]
                r.finished = now
                if status[tick_index[id(s)]] & bad:
                    r.error = "NaN detected in MPM states"
                    if not s.retired:  # evict it from the current layout
                        self._retire(next(k for k, o in enumerate(self.active) if o is s))
                elif id(s) in fin_host:
                    r.pos, r.vel = (t.numpy() for t in fin_host[id(s)])
                if on_result is not None:
                    on_result(r)
        self.rt = None
        self.active = []
        return [results[r.rid] for r in reqs]


def percentile(xs, q):
    xs = sorted(x for x in xs if x is not None)
    if not xs:
        return None
    k = (len(xs) - 1) * q / 100.0
    f, c = math.floor(k), math.ceil(k)
    return xs[f] if f == c else xs[f] + (xs[c] - xs[f]) * (k - f)


def sequential_timeline(requests, durations):
    """Latencies of the plain one-request-at-a-time path under the same arrivals: each
    request starts when it has arrived and the previous one has finished."""
    t = 0.0
    lat = []
    for r, d in sorted(zip(requests, durations), key=lambda x: x[0].arrival):
        start = max(t, r.arrival)
        t = start + d
        lat.append(t - r.arrival)
    return lat
