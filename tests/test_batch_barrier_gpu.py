"""A grid barrier of the batched engine's resident step kernel that runs out.

The barrier is the real one, given no time to wait: every block but the last to arrive gives up and
returns. No fault is provoked. Reading then fails, and so do stepping and admitting from then on; once
every instance is retired the batch steps new ones as a fresh batch does.
"""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [32, 64])
def test_barrier_runs_out_and_the_batch_recovers(precision):
    if not torch.cuda.is_available():
        pytest.fail("CUDA GPU required for -m gpu tests")
    from tensordem_gb300 import _lib, batch as bt
    insts = [s.build() for s in bt.ensemble_case(4, seed=2, n_min=100, n_max=900, steps=400)]
    cfg = bt.BatchConfig(particle_capacity=sum(i.n for i in insts) + 64, key_capacity=sum(i.keys for i in insts) + 64,
                         max_instances=8, precision=precision)
    b, fresh = bt.Batch(cfg), bt.Batch(cfg)
    ids = [b.admit(i) for i in insts]
    b.step(3)
    b.ledgers(ids)
    assert _lib.lib().tdem_batch_set_wait_budget(b._h, -1) != 0
    assert _lib.lib().tdem_batch_set_wait_budget(b._h, 0) == 0
    b.step(5)
    for call in (lambda: b.bonds(ids[0]), lambda: b.read(ids[1]), lambda: b.ledgers(ids), lambda: b.step(1),
                 lambda: b.admit(insts[0])):
        with pytest.raises(RuntimeError, match="bounded wait"):
            call()
    assert b.info()["status"] & 16
    assert _lib.lib().tdem_batch_set_wait_budget(b._h, 2_000_000_000) == 0
    for k in ids:
        with pytest.raises(RuntimeError, match="bounded wait"):
            b.step(1)
        b.retire(k)
    b.step(0)   # the compaction that frees their places
    again, want = [b.admit(i) for i in insts], [fresh.admit(i) for i in insts]
    for x in (b, fresh):
        x.step(1)
        x.step(24)
    assert b.info()["status"] == 0
    for i, j, inst in zip(again, want, insts):
        x, y = b.read(i), fresh.read(j)
        for k in ("pos", "vel", "omega", "force", "torque"):
            assert np.array_equal(x[k], y[k]), k
        skip = ("rebuilds", "graph")
        assert {k: v for k, v in x["ledger"].items() if k not in skip} == \
            {k: v for k, v in y["ledger"].items() if k not in skip}
        if inst.bonds is not None:
            p, q = b.bonds(i), fresh.bonds(j)
            assert all(np.array_equal(p[k], q[k]) for k in p)
