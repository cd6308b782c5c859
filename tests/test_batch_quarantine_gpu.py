"""An instance that goes non-finite in the batched engine's resident step loop.

The evaluation in which it happens belongs to the instance as a whole: every tile takes it and its
ledger row is booked once, whichever warp comes to which tile first; from the next evaluation on the
instance is frozen. The instance here fills several warps behind a large one, with a warp in between
that reaches its first tile last, after another warp has met the bad disc in the second tile.
"""

from dataclasses import replace

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

COLUMNS = 32   # discs of a row: one cell each, so row k of an instance is its tile k


@pytest.fixture(scope="module")
def bt():
    if not torch.cuda.is_available():
        pytest.fail("CUDA GPU required for -m gpu tests")
    from tensordem_gb300 import batch
    return batch


def _rows(bt, rows, precision, seed):
    """A dilute instance of `rows` tiles whose indenter touches nothing."""
    from tensordem_gb300.hm2d import HM2DConfig
    n = rows * COLUMNS
    jj, ii = np.meshgrid(np.arange(rows), np.arange(COLUMNS), indexing="ij")
    pos = np.stack((ii.ravel() + 0.5, jj.ravel() + 0.5), axis=1)
    vel = np.random.default_rng(seed).normal(0.0, 0.01, (n, 2))
    radius, mass = np.full(n, 0.3), np.ones(n)
    cfg = HM2DConfig(n=n, ncx=COLUMNS, ncy=rows, cell=1.0, skin=0.2, dt=2e-4, young=1e9, poisson=0.3, restitution=0.8,
                     mu=0.3, mu_wall=0.3, gravity=(0.0, 0.0), precision=precision, indenter_center=(-1e3, -1e3),
                     indenter_velocity=(0.0, -0.01), indenter_radius=0.05)
    state = dict(pos=pos, vel=vel, omega=np.zeros(n), radius=radius, mass=mass, inertia=0.5 * mass * radius**2)
    return bt.Instance(cfg, state)


def _failing(bt, rows, precision):
    """The same with the indenter on a heavy disc of tile 0 and two overlapping discs in tile 3; in tile 1
    a disc so light that its first contact, after five steps, overflows its acceleration."""
    inst = _rows(bt, rows, precision, 5)
    s = inst.state
    s["mass"][10] = 1e3
    s["vel"][10] = 0.0
    s["pos"][3 * COLUMNS + 7, 0] += 0.401                    # overlaps its right neighbour by 1e-3
    light = COLUMNS + 4
    s["mass"][light] = 1e-37 if precision == 32 else 1e-307
    s["pos"][light, 0] += 0.4 - 1.1e-3                       # 1.1e-3 from its right neighbour
    s["vel"][light:light + 2] = ((1.0, 0.0), (0.0, 0.0))
    s["inertia"] = 0.5 * s["mass"] * s["radius"]**2
    x, y = s["pos"][10]
    inst.config = replace(inst.config, indenter_center=(x, y + 0.35 - 1e-3))
    return inst


def _run(bt, insts, precision, graph=True, steps=20):
    b = bt.Batch(bt.BatchConfig(particle_capacity=sum(i.n for i in insts) + 64,
                                key_capacity=sum(i.keys for i in insts) + 64, max_instances=4, precision=precision,
                                max_bonds=0))
    b.use_graph(graph)
    ids = [b.admit(i) for i in insts]
    b.step(steps)
    led = b.ledgers(ids)
    return b.read(ids[0]), [{k: r[k] for k in ("dissipated", "tool_work", "broken", "peak_load", "peak_eval",
                                               "reaction_x", "reaction_y", "status")} for r in led]


@pytest.mark.parametrize("precision", [32, 64])
def test_the_evaluation_that_goes_non_finite_is_booked_whole(bt, precision):
    warps = torch.cuda.get_device_properties(0).multi_processor_count * (16 if precision == 32 else 8)
    rows = 100
    other = _rows(bt, 3 * warps - rows, precision, 3)        # three tiles a warp
    assert (3 * warps - rows) % 3 == 2                       # one warp: two of its tiles, then tile 0 of the failing one
    failing = _failing(bt, rows, precision)
    state, (_, got) = _run(bt, [other, failing], precision)
    _, (alone,) = _run(bt, [failing], precision)             # a tile a warp: all meet it at once
    assert int(alone["status"]) & 2 and alone["tool_work"] > 0.0 and alone["peak_load"] > 0.0
    before, (early,) = _run(bt, [failing], precision, steps=5)
    assert int(early["status"]) == 0 and early["tool_work"] < alone["tool_work"] and early["dissipated"] != 0.0
    assert got == alone
    # the other instance is as in the one-step kernels
    plain, _ = _run(bt, [other, failing], precision, graph=False)
    for k in ("pos", "vel", "omega", "force", "torque"):
        assert np.array_equal(state[k], plain[k]), k
