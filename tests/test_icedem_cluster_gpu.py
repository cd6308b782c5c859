"""Reference mode over a thread-block cluster against the FP64 oracle, at the shapes where the
deal of the discs can go wrong: a CTA with one disc, CTAs without any, partial groups, several
rounds of discs per warp, and the largest lattice (one copy of the positions); and a heap of
overlapping discs with more force terms than a disc's list holds.

The oracle sums the same terms in the same order; 1e-12 is the suite's bound for reference
mode (a few roundings of torch-free square roots and divisions apart at most).
"""

import numpy as np
import pytest
import torch

from oracle.icedem import IceDEMOracle, OracleConfig

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tdem():
    if not torch.cuda.is_available():
        pytest.fail("CUDA GPU required for -m gpu tests")
    import tensordem_gb300
    return tensordem_gb300


def _close(a, b, scale=None):
    a, b = np.asarray(a, dtype=np.float64), np.asarray(b, dtype=np.float64)
    assert np.abs(a - b).max() <= 1e-12 * max(1e-300, np.abs(b).max() if scale is None else scale)


@pytest.mark.parametrize("nx,ny,steps", [(2, 2, 40), (3, 2, 40), (6, 3, 40), (13, 5, 40), (37, 11, 12), (64, 32, 3)])
def test_steps_equal_the_oracle(tdem, nx, ny, steps):
    kw = dict(nx=nx, ny=ny, tool_speed=0.5, breaking_strain=1e-3, shear_breaking_strain=2e-3)
    gpu = tdem.IceDEM(tdem.DEMConfig(**kw))
    cpu = IceDEMOracle(OracleConfig(**kw))
    rng = np.random.default_rng(nx * ny)
    v = rng.normal(0.0, 0.5, cpu.velocities.shape)
    v[cpu.fixed] = 0.0
    cpu.velocities = v.copy()
    gpu.velocities = torch.from_numpy(v).to(gpu.device)
    load = rng.normal(0.0, 1.0, v.shape)
    gpu.run(steps - 1)
    gpu.step(torch.from_numpy(load).to(gpu.device))
    for _ in range(steps - 1):
        cpu.step()
    cpu.step(load)
    _close(gpu.positions.cpu(), cpu.positions)
    _close(gpu.velocities.cpu(), cpu.velocities)
    assert np.array_equal(gpu.alive.cpu().numpy(), cpu.alive)
    assert np.array_equal(gpu.failure_mode.cpu().numpy(), cpu.failure_mode)
    f, r = gpu.forces()
    fc, rc = cpu.forces()
    _close(f.cpu(), fc)
    _close(r.cpu(), rc, max(1.0, np.abs(fc).max()))
    acc = gpu.accounting
    scale = max(abs(x) for x in (acc["damping_dissipation_J"], acc["fracture_release_J"], 1e-9))
    for key in cpu.LEDGER_KEYS:
        _close(acc[key], cpu.accounting[key], scale)
    for key in cpu.IMPULSE_KEYS:
        _close(acc[key], cpu.accounting[key], max(1e-9, np.abs(np.asarray(acc["drag_impulse_Ns"])).max()))


def test_a_heap_with_more_terms_than_the_lists_hold(tdem):
    kw = dict(nx=12, ny=8, fix_edges=False)
    gpu = tdem.IceDEM(tdem.DEMConfig(**kw))
    cpu = IceDEMOracle(OracleConfig(**kw))
    rng = np.random.default_rng(4)
    r = gpu.config.radius
    pos = rng.uniform(-3.0 * r, 3.0 * r, cpu.positions.shape)   # a third of the pairs overlap
    vel = rng.normal(0.0, 0.1, pos.shape)
    keep = rng.uniform(size=cpu.alive.shape) < 0.5               # half of the bonds already broken
    for sim, t in ((cpu, lambda a: a), (gpu, lambda a: torch.from_numpy(a).to(gpu.device))):
        sim.positions, sim.velocities = t(pos.copy()), t(vel.copy())
    cpu.alive &= keep
    gpu.alive = torch.from_numpy(cpu.alive.copy()).to(gpu.device)
    gpu.failure_mode[gpu.bonded & ~gpu.alive] = 1
    near = (np.sqrt(((pos[:, None] - pos[None]) ** 2).sum(2)) < 2 * r).sum(1) - 1
    assert near.max() > 32 and near.min() < 32
    f, _ = gpu.forces()
    fc, _ = cpu.forces()
    _close(f.cpu(), fc)
    assert np.array_equal(gpu.alive.cpu().numpy(), cpu.alive)
