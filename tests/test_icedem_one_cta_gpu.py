"""The reference mode's one-CTA kernel, which steps discs of more than eight bonds, against the FP64 oracle.

The Python surface builds square lattices (eight bonds a disc at most); here the native engine gets one
whose spacing is 1.4 radii, so that an inner disc has twelve, with the tool pressed into it, bonds that
break, nodal loads and (once) per-bond stiffnesses. 1e-12 is the suite's bound for reference mode.
"""

import ctypes as C
import math

import numpy as np
import pytest
import torch

from oracle.icedem import IceDEMOracle, OracleConfig, vnorm2

pytestmark = pytest.mark.gpu


def _close(a, b, scale=None):
    a, b = np.asarray(a, dtype=np.float64), np.asarray(b, dtype=np.float64)
    assert np.abs(a - b).max() <= 1e-12 * max(1e-300, np.abs(b).max() if scale is None else scale)


def _pair(kw, x0):
    """Oracle and engine on the lattice x0."""
    import tensordem_gb300 as tdem
    cpu = IceDEMOracle(OracleConfig(**kw))
    cpu.positions, cpu.initial_positions = x0.copy(), x0.copy()
    i, j = cpu.pairs.T
    delta = x0[j] - x0[i]
    cpu.rest_lengths = vnorm2(delta)
    cpu.initial_normals = delta / cpu.rest_lengths[:, None]
    cpu.bonded = cpu.rest_lengths <= 2 * cpu.config.radius * math.sqrt(2) * (1 + 1e-10)
    cpu.bond_indices = cpu.pairs[cpu.bonded]
    cpu.reference_bond_vectors = delta[cpu.bonded]
    cpu.alive = cpu.bonded.copy()
    gpu = tdem.IceDEM(tdem.DEMConfig(**kw))
    gpu.initial_positions = torch.from_numpy(x0.copy()).to(gpu.device)
    gpu.positions = gpu.initial_positions.clone()
    gpu._build_native()
    gpu.bonded = torch.from_numpy(cpu.bonded.copy()).to(gpu.device)
    gpu.alive = gpu.bonded.clone()
    assert np.array_equal(np.flatnonzero(cpu.bonded), gpu._bond_pair_index.numpy())
    return cpu, gpu


@pytest.mark.parametrize("nx,ny,steps,stiffness", [(5, 5, 4, False), (9, 7, 8, False), (9, 7, 8, True),
                                                   (31, 20, 14, False)])
def test_twelve_bonds_a_disc(nx, ny, steps, stiffness):
    if not torch.cuda.is_available():
        pytest.fail("CUDA GPU required for -m gpu tests")
    from tensordem_gb300 import _lib
    kw = dict(nx=nx, ny=ny, tool_speed=0.5, breaking_strain=2e-4, shear_breaking_strain=4e-4)
    r = OracleConfig().radius
    yy, xx = np.meshgrid(np.arange(ny, dtype=float), np.arange(nx, dtype=float), indexing="ij")
    x0 = np.stack((xx.ravel() - (nx - 1) / 2, yy.ravel()), axis=1) * (1.4 * r)
    x0[:, 1] += 0.6 * r * (ny - 1) + 0.01 + 1e-5   # the tool is 1e-5 m in the top row
    cpu, gpu = _pair(kw, x0)
    degree = np.bincount(cpu.bond_indices.ravel(), minlength=nx * ny)
    assert degree.max() > 8
    rng = np.random.default_rng(nx)
    if stiffness:
        k = rng.uniform(0.5, 1.0, len(cpu.bond_indices)) * cpu.config.bond_stiffness
        cpu.pair_coefficients = np.zeros(len(cpu.pairs))
        cpu.pair_coefficients[cpu.bonded] = k
        rc = _lib.lib().tdem_icedem_set_bond_stiffness(gpu._handle.ptr, C.cast(k.ctypes.data, C.POINTER(C.c_double)),
                                                       len(k))
        assert rc == 0
    v = rng.normal(0.0, 0.02, x0.shape)
    v[cpu.fixed] = 0.0
    cpu.velocities = v.copy()
    gpu.velocities = torch.from_numpy(v).to(gpu.device)
    load = rng.normal(0.0, 1.0, v.shape)
    gpu.run(steps - 1)
    gpu.step(torch.from_numpy(load).to(gpu.device))
    for _ in range(steps - 1):
        cpu.step()
    cpu.step(load)
    assert 0 < cpu.broken_bonds < cpu.bonded.sum()
    _close(gpu.positions.cpu(), cpu.positions)
    _close(gpu.velocities.cpu(), cpu.velocities)
    assert np.array_equal(gpu.alive.cpu().numpy(), cpu.alive)
    assert np.array_equal(gpu.failure_mode.cpu().numpy(), cpu.failure_mode)
    f, reaction = gpu.forces()
    fc, rc = cpu.forces()
    _close(f.cpu(), fc)
    _close(reaction.cpu(), rc, max(1.0, np.abs(fc).max()))
    acc = gpu.accounting
    assert abs(acc["tool_work_J"]) > 0.0
    scale = max(abs(x) for x in (acc["damping_dissipation_J"], acc["fracture_release_J"], 1e-9))
    for key in cpu.LEDGER_KEYS:
        _close(acc[key], cpu.accounting[key], scale)
    for key in cpu.IMPULSE_KEYS:
        _close(acc[key], cpu.accounting[key], max(1e-9, np.abs(np.asarray(acc["drag_impulse_Ns"])).max()))
    last = gpu.last_step
    assert (last["time_start_s"], last["time_end_s"]) == (cpu.last_step["time_start_s"], cpu.last_step["time_end_s"])
