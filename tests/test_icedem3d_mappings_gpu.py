"""The 3-D step's lane mappings at their edges: specimens around the particle count from which the
shear takes four lanes a particle instead of sixteen (2,432 on 152 SMs), counts that are no multiple
of the sixteen particles whose pairs a warp takes together, and a specimen of few particles with many
contacts. Every mapping must give the one-thread-per-particle step's bits.
"""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(mapping, size, squeeze, seed, **kw):
    from tensordem_gb300.dem3d import DEM3DConfig, IceDEM3D
    sim = IceDEM3D(DEM3DConfig(nx=size[0], ny=size[1], nz=size[2], breaking_strain=0.004,
                               shear_breaking_strain=0.008, restitution_coefficient=0.7, **kw))
    sim.set_thread_mapping(mapping)
    rng = np.random.default_rng(seed)
    v = torch.from_numpy(rng.normal(0.0, 0.5, tuple(sim.positions.shape))).to(sim.device)
    v[sim.fixed] = 0.0
    sim.velocities = v
    if squeeze:   # overlapping neighbours, most bonds broken
        sim.positions = sim.positions * 0.97
    sim.run(40)
    return sim


@pytest.mark.parametrize("size,squeeze,kw", [
    ((5, 3, 2), True, dict(friction_coefficient=0.3, rolling_resistance_coefficient=0.1)),
    ((9, 7, 5), True, dict(friction_coefficient=0.3, contact_model="hertz")),
    ((20, 15, 8), False, dict(friction_coefficient=0.3)),     # 2,400: sixteen lanes
    ((17, 16, 9), False, dict(friction_coefficient=0.3)),     # 2,448: four lanes
    ((31, 11, 9), True, dict()),
])
def test_mappings_give_the_same_bits(size, squeeze, kw):
    a, b = _run("lanes", size, squeeze, 7, **kw), _run("particle", size, squeeze, 7, **kw)
    for name in ("positions", "velocities", "alive", "failure_mode", "failure_time_s", "failure_extension_m"):
        assert torch.equal(getattr(a, name), getattr(b, name)), name
    assert a.friction_history() == b.friction_history()
    assert a.broken_bonds > 0 and torch.equal(a.contact_pairs(), b.contact_pairs())
    # ledger sums combine the same terms per thread of another shape: rounding only
    la, lb = a.read_ledger(), b.read_ledger()
    assert np.allclose(la, lb, rtol=1e-12, atol=1e-12 * max(1.0, np.abs(lb[np.abs(lb) < 1e299]).max()))
