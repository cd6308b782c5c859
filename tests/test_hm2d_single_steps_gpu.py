"""Single steps beside blocks of steps: ``step(1)`` has a graph of its own.

Small FP32 engines and the pipelined variants take the one-step kernel there, FP64 engines and large
FP32 ones one evaluation of the resident kernel, and both go on where blocks of resident steps end
(and the other way round): states, histories, bonds and ledgers must be those of plain launches bit
for bit. A state's first single step is plain launches, which a user's stream capture takes.
"""

import pytest
import torch

from tests._hm_cases import dense_gas, small_sheet
from tests.test_hm2d_resident_gpu import _run, _same

pytestmark = pytest.mark.gpu

BLOCKS = (1, 1, 5, 1, 1, 1, 30, 1, 2, 1)


@pytest.fixture(scope="module")
def hm():
    if not torch.cuda.is_available():
        pytest.fail("CUDA GPU required for -m gpu tests")
    from tensordem_gb300 import hm2d
    return hm2d


def _engine(hm, cfg, st, bonds, graph, variant):
    if variant == 0:
        return _run(hm, cfg, st, bonds, graph, BLOCKS)
    e = hm.HM2D(cfg)
    e.use_graph(graph)
    e.variant = variant
    e.set_state(st["pos"], st["vel"], st["omega"], st["radius"], st["mass"], st["inertia"])
    if bonds is not None:
        e.set_bonds(*bonds)
    for n in BLOCKS:
        e.step(n)
    return e


# one block, a grid with a thread per pair, more discs than threads (pipelined, default variant and 10), FP64
@pytest.mark.parametrize("precision,side,variant", [(32, 22, 0), (32, 57, 0), (32, 400, 0), (32, 400, 10), (64, 57, 0)])
def test_granular_single_steps_among_blocks(hm, precision, side, variant):
    cfg, st = dense_gas(side, seed=side, precision=precision, skin=0.5e-3)
    a = _engine(hm, cfg, st, None, True, variant)
    led = _same(a, _engine(hm, cfg, st, None, False, variant), False)
    assert led["evals"] == sum(BLOCKS) and led["status"] == 0


@pytest.mark.parametrize("precision,nx,ny,variant", [(32, 26, 7, 0), (32, 400, 200, 0), (32, 80, 40, 11), (64, 61, 13, 0)])
def test_bonded_single_steps_among_blocks(hm, precision, nx, ny, variant):
    cfg, st, bonds, strength = small_sheet(nx, ny, precision=precision, steps=400, speed=20.0)
    a = _engine(hm, cfg, st, (bonds, strength), True, variant)
    led = _same(a, _engine(hm, cfg, st, (bonds, strength), False, variant), True)
    assert led["evals"] == sum(BLOCKS) and led["tool_work"] > 0.0


def test_a_first_single_step_builds_no_graph_and_can_be_captured(hm):
    cfg, st = dense_gas(40, seed=3)

    def fresh():
        e = hm.HM2D(cfg)
        e.set_state(st["pos"], st["vel"], st["omega"], st["radius"], st["mass"], st["inertia"])
        return e
    plain, captured = fresh(), fresh()
    plain.step(1)
    assert not plain.ledger()["graph"]
    captured.anchor   # the torch op's device argument
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        captured.step(1, check=False)
    g.replay()
    torch.cuda.synchronize()
    captured.check()
    captured.step(20)
    plain.step(20)
    _same(captured, plain, False)
