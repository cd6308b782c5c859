"""The batched engine's resident step kernel (the default step loop) against its one-step kernels.

The same tiles are evaluated by the same code, so states, bonds and ledgers must be equal
bit for bit: a few tiles (most warps of the grid idle), more tiles than warps, instances
that reach their step limit, retire and join between blocks, and list rebuilds.
"""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def bt():
    if not torch.cuda.is_available():
        pytest.fail("CUDA GPU required for -m gpu tests")
    from tensordem_gb300 import batch
    return batch


def _drive(bt, insts, late, precision, graph, remainder, every):
    cfg = bt.BatchConfig(particle_capacity=sum(i.n for i in insts) + late.n + 64,
                         key_capacity=sum(i.keys for i in insts) + late.keys + 64, max_instances=64,
                         precision=precision, position_remainder=remainder, rebuild_every=every)
    b = bt.Batch(cfg)
    b.use_graph(graph)
    ids = [b.admit(i) for i in insts]
    b.set_steps(ids[1], 5)
    b.step(1)
    b.step(7)
    b.retire(ids[2])
    ids[2] = b.admit(late)
    b.step(40)
    out = [b.read(k) for k in ids]
    bonds = [b.bonds(k) for k, i in zip(ids, insts[:2] + [late] + insts[3:]) if i.bonds is not None]
    return out, b.ledgers(ids), bonds, b.info()


@pytest.mark.parametrize("runs,n_max,precision,remainder,every",
                         [(5, 200, 32, 1, 0), (5, 200, 64, 1, 0), (40, 9000, 32, 1, 20), (24, 3000, 32, 0, 0),
                          (30, 9000, 64, 1, 20)])
def test_resident_steps_equal_one_step_launches(bt, runs, n_max, precision, remainder, every):
    insts = [s.build() for s in bt.ensemble_case(runs + 1, seed=9, n_min=100, n_max=n_max, steps=400)]
    for i in insts:   # residual motion, so that bonds, contacts and walls are at work
        vel = np.random.default_rng(i.n).normal(0.0, 0.3, i.state["pos"].shape)
        vel[~np.isfinite(i.state["mass"])] = 0.0
        i.state["vel"] = vel
    a = _drive(bt, insts[:-1], insts[-1], precision, True, remainder, every)
    b = _drive(bt, insts[:-1], insts[-1], precision, False, remainder, every)
    for x, y in zip(a[0], b[0]):
        for k in ("pos", "vel", "omega", "force", "torque"):
            assert np.array_equal(x[k], y[k]), k
    skip = ("graph",)
    for x, y in zip(a[1], b[1]):
        assert {k: v for k, v in x.items() if k not in skip} == {k: v for k, v in y.items() if k not in skip}
    assert all(np.array_equal(x[k], y[k]) for x, y in zip(a[2], b[2]) for k in x)
    assert a[3]["graph"] == 1 and a[3]["evals"] == 48 and a[3]["rebuilds"] == b[3]["rebuilds"]
    assert a[1][1]["evals"] == 5   # the limited instance stopped
