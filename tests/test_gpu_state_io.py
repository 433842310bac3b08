"""State written and read back through the staged row copies, at sizes around a warp and a CTA, in API
order while the particles are sorted: every bit comes back, whole and by parts."""

import numpy as np
import pytest
import torch

from genesis_b200 import workloads as W
from genesis_b200.engine.runtime import runtime_from_descs


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 31, 32, 33, 255, 257, 1000])
def test_state_comes_back_bit_for_bit(n):
    d = W.elastic_cube(n_side=10)
    d.pos, d.vel, d.mat_idx = d.pos[:n], d.vel[:n], d.mat_idx[:n]
    rt = runtime_from_descs([d])
    rt.sort()
    g = torch.Generator(device="cuda").manual_seed(n)
    want = {"pos": torch.as_tensor(d.pos, dtype=torch.float32, device="cuda"),
            "vel": torch.randn((n, 3), generator=g, device="cuda"), "C": torch.randn((n, 3, 3), generator=g, device="cuda"),
            "F": torch.randn((n, 3, 3), generator=g, device="cuda"), "Jp": torch.randn(n, generator=g, device="cuda"),
            "active": torch.arange(n, device="cuda") % 3 != 1}
    rt.set_state(want["pos"], want["vel"], want["C"], want["F"], want["Jp"], want["active"])
    rt.sort()  # another slot order
    got = rt.get_state()
    for k, v in want.items():
        assert torch.equal(got[k], v), k
    F2 = torch.randn((n, 3, 3), generator=g, device="cuda")
    rt.set_state(F=F2)
    got = rt.get_state(("F", "C"))
    assert torch.equal(got["F"], F2) and torch.equal(got["C"], want["C"]) and set(got) == {"F", "C"}
    assert np.array_equal(np.sort(rt.gid[:n].cpu().numpy()), np.arange(n))
