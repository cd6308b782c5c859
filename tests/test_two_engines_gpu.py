"""Several engines at once, each driven by a host thread on a stream of its own.

The resident kernels are cooperative grids of up to one block per SM (the reference mode a cluster of
16), so engines on other streams wait for room: each must still give the bits that it gives alone.
"""

import threading

import numpy as np
import pytest
import torch

from tests._hm_cases import dense_gas, small_sheet

pytestmark = pytest.mark.gpu


def _discs(side, precision=32, variant=0):
    from tensordem_gb300.hm2d import HM2D
    cfg, st = dense_gas(side, seed=side, precision=precision, skin=0.5e-3)
    e = HM2D(cfg)
    e.variant = variant

    def drive():
        e.set_state(st["pos"], st["vel"], st["omega"], st["radius"], st["mass"], st["inertia"])
        for n in (1, 30, 1, 40, 29):
            e.step(n)
        return {k: t.cpu().numpy() for k, t in e.state().items()}
    return drive


def _sheet(nx, ny):
    from tensordem_gb300.hm2d import HM2D
    cfg, st, *bonds = small_sheet(nx, ny, precision=32, steps=400, speed=20.0)
    e = HM2D(cfg)

    def drive():
        e.set_state(st["pos"], st["vel"], st["omega"], st["radius"], st["mass"], st["inertia"])
        e.set_bonds(*bonds)
        for n in (50, 1, 99):
            e.step(n)
        return {k: t.cpu().numpy() for k, t in e.state().items()}
    return drive


def _batch(runs):
    from tensordem_gb300 import batch as bt
    insts = [s.build() for s in bt.ensemble_case(runs, seed=9, n_min=100, n_max=900, steps=400)]
    cfg = bt.BatchConfig(particle_capacity=sum(i.n for i in insts) + 64, key_capacity=sum(i.keys for i in insts) + 64,
                         max_instances=runs)

    def drive():
        b = bt.Batch(cfg)
        ids = [b.admit(i) for i in insts]
        for _ in range(4):
            b.step(25)
        out = [b.read(k) for k in ids]
        return {f"{k}{q}": row[k] for q, row in enumerate(out) for k in ("pos", "vel", "omega", "force", "torque")}
    return drive


def _lattice():
    import tensordem_gb300 as tdem

    def drive():
        sim = tdem.IceDEM(tdem.DEMConfig(nx=21, ny=5, tool_speed=0.5, breaking_strain=1e-3, shear_breaking_strain=2e-3))
        for _ in range(4):
            sim.run(25)
        return dict(pos=sim.positions.cpu().numpy(), vel=sim.velocities.cpu().numpy(), alive=sim.alive.cpu().numpy())
    return drive


def _specimen():
    from tensordem_gb300.dem3d import DEM3DConfig, IceDEM3D

    def drive():
        sim = IceDEM3D(DEM3DConfig(nx=20, ny=10, nz=6, breaking_strain=0.004, shear_breaking_strain=0.008))
        for _ in range(4):
            sim.run(10)
        return dict(pos=sim.positions.cpu().numpy(), vel=sim.velocities.cpu().numpy(), alive=sim.alive.cpu().numpy())
    return drive


@pytest.mark.parametrize("makers", [
    [lambda: _discs(230), lambda: _discs(240)],                     # two grids of most of the chip
    [lambda: _discs(400), lambda: _discs(400, variant=10)],         # two pipelined grids of all of it
    [lambda: _discs(100, precision=64), lambda: _sheet(80, 40), lambda: _batch(8)],
    [lambda: _discs(57), lambda: _batch(8), lambda: _lattice(), lambda: _specimen()],
])
def test_engines_on_streams_of_their_own(makers):
    if not torch.cuda.is_available():
        pytest.fail("CUDA GPU required for -m gpu tests")
    drives = [m() for m in makers]
    alone = [d() for d in drives]
    got, errors = [None] * len(drives), []

    def work(k):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(3):
                    got[k] = drives[k]()
        except Exception as e:  # noqa: BLE001  (re-raised below)
            errors.append(e)
    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(drives))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for a, b in zip(alone, got):
        for k in a:
            assert np.array_equal(a[k], b[k]), k
