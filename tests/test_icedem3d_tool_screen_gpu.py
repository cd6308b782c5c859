"""The FP32 screen of the 3-D step's tool contact (several lanes a particle) drops no contact, also at
sizes whose squares underflow in FP32: the step with one thread a particle has no screen.
"""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radius", [2e-23, 1e-19, 0.025])
def test_contacts_at_the_edge_of_reach(radius):
    if not torch.cuda.is_available():
        pytest.fail("CUDA GPU required for -m gpu tests")
    from tensordem_gb300.dem3d import DEM3DConfig, IceDEM3D
    cfg = DEM3DConfig(nx=2, ny=2, nz=2, radius=radius, tool_radius=4 * radius, tool_gap=0.0)
    sims = {}
    for mapping in ("lanes", "particle"):
        sims[mapping] = IceDEM3D(cfg)
        sims[mapping].set_thread_mapping(mapping)
    rng = np.random.default_rng(1)
    tool = sims["lanes"].tool_start.cpu().numpy()
    touched = 0
    for _ in range(100):
        d = rng.normal(size=(8, 3))
        d *= (5 * radius * rng.uniform(0.9, 1.02, 8) / np.sqrt((d**2).sum(1)))[:, None]
        out = []
        for sim in sims.values():
            sim.positions = torch.from_numpy(tool + d).to(sim.device)
            sim.alive = torch.zeros_like(sim.alive)
            force, reaction = sim.forces()
            out.append((force, reaction))
        assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
        touched += int((out[1][1] != 0).any())
    assert touched > 90
