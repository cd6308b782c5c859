"""The resident step kernel (the default step loop) against the one-step kernels.

Both run the same per-disc code in the same order, so the states, bonds and
ledgers must be equal bit for bit, whatever the block shape: one block, its
edge, partial last blocks, the build for engines that need every thread of the
chip, and engines too large for it. Lists are rebuilt on the way, and steps
come in blocks of one and of many.
"""

import numpy as np
import pytest
import torch

from tests._hm_cases import dense_gas, small_sheet

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def hm():
    if not torch.cuda.is_available():
        pytest.fail("CUDA GPU required for -m gpu tests")
    from tensordem_gb300 import hm2d
    return hm2d


def _run(hm, cfg, st, bonds, graph, blocks):
    e = hm.HM2D(cfg)
    e.use_graph(graph)
    e.set_state(st["pos"], st["vel"], st["omega"], st["radius"], st["mass"], st["inertia"])
    if bonds is not None:
        e.set_bonds(*bonds)
    for n in blocks:
        e.step(n)
    return e


def _same(a, b, bonded):
    for k, x in a.state().items():
        assert torch.equal(x, b.state()[k]), k
    la, lb = a.ledger(), b.ledger()
    for k in ("dissipated", "total", "evals", "rebuilds", "bond_elastic", "fracture_released", "tool_work", "broken"):
        assert la[k] == lb[k], (k, la[k], lb[k])
    assert a.history() == b.history()
    if bonded:
        ba, bb = a.bonds(), b.bonds()
        assert all(np.array_equal(ba[k], bb[k]) for k in ba)
        assert np.array_equal(a.load_curve(), b.load_curve())
    return la


# 4 and 484 discs: one block; 529: the first grid; 3249: a partial last block; 80089: the big
# build (FP64: too large); 160000: more discs than threads. The narrow skin leaves under one
# candidate pair per disc (a thread per disc), the wide one more (a thread per pair).
@pytest.mark.parametrize("skin", [0.02e-3, 0.5e-3])
@pytest.mark.parametrize("precision,side", [(32, 2), (32, 22), (32, 23), (32, 57), (32, 283), (32, 400),
                                            (64, 16), (64, 33), (64, 205), (64, 283)])
def test_granular_resident_steps_equal_one_step_launches(hm, precision, side, skin):
    cfg, st = dense_gas(side, seed=side, precision=precision, skin=skin)
    blocks = (1, 2, 1, 60)
    a = _run(hm, cfg, st, None, True, blocks)
    led = _same(a, _run(hm, cfg, st, None, False, blocks), False)
    assert led["evals"] == 64 and led["status"] == 0
    if side >= 22:
        assert led["dissipated"] > 0.0 and (led["rebuilds"] >= 2 or skin > 0.1e-3)


# 90 and 128 discs: one block; 182: the first grid; 40000: the big build (FP64 too)
@pytest.mark.parametrize("precision,nx,ny", [(32, 15, 6), (32, 16, 8), (32, 26, 7), (32, 80, 40), (32, 400, 100),
                                             (64, 15, 6), (64, 61, 13), (64, 400, 100)])
def test_bonded_resident_steps_equal_one_step_launches(hm, precision, nx, ny):
    cfg, st, bonds, strength = small_sheet(nx, ny, precision=precision, steps=400, speed=20.0)
    blocks = (1, 3, 196)
    a = _run(hm, cfg, st, (bonds, strength), True, blocks)
    led = _same(a, _run(hm, cfg, st, (bonds, strength), False, blocks), True)
    assert led["evals"] == 200 and led["tool_work"] > 0.0


# wide skins: more pairs per disc than a block's shared memory holds, so its threads work on
# the global arrays (FP32 and FP64 big builds)
@pytest.mark.parametrize("precision,side,skin,slots", [(32, 390, 2.0e-3, 24), (64, 277, 2.5e-3, 24)])
def test_blocks_without_room_for_their_pairs(hm, precision, side, skin, slots):
    cfg, st = dense_gas(side, seed=side, precision=precision, skin=skin, max_neighbors=slots)
    a = _run(hm, cfg, st, None, True, (25,))
    led = _same(a, _run(hm, cfg, st, None, False, (25,)), False)
    assert led["status"] == 0 and led["dissipated"] > 0.0


# pairs per disc of a block (2.0, 3.6 and 4.0, and those that two blocks evaluate) on both sides
# of the two thirds of its room (6.2) up to which FP64 pairs keep their effective radius and mass
@pytest.mark.parametrize("skin", [0.5e-3, 1.0e-3, 1.5e-3])
def test_fp64_pairs_with_and_without_room_for_their_constants(hm, skin):
    cfg, st = dense_gas(270, seed=270, precision=64, skin=skin, max_neighbors=24)
    a = _run(hm, cfg, st, None, True, (1, 40))
    led = _same(a, _run(hm, cfg, st, None, False, (1, 40)), False)
    assert led["status"] == 0 and led["dissipated"] > 0.0


# one block up to 4096 discs (FP64 512, bonded 1024, FP64 bonded 128) rebuilds the lists of a small
# grid; the same discs in a corner of a grid of 40,000 cells sort alike and take the general pipeline
@pytest.mark.parametrize("precision,side,nx,ny", [(32, 3, 0, 0), (32, 40, 0, 0), (32, 64, 0, 0), (64, 22, 0, 0),
                                                  (32, 0, 24, 8), (32, 0, 64, 16), (64, 0, 12, 8)])
def test_one_block_rebuild_equals_the_general_one(hm, precision, side, nx, ny):
    from dataclasses import replace
    if side:
        cfg, st = dense_gas(side, seed=side, precision=precision, walls=5, sigma_v=8.0)
        bonds, blocks = None, (1, 200)
    else:
        cfg, st, *bonds = small_sheet(nx, ny, precision=precision, steps=400, speed=20.0)
        blocks = (1, 199)
    small = replace(cfg, ncx=cfg.ncx + 2, ncy=cfg.ncy + 2)
    assert -(-small.ncx // 32) * -(-small.ncy // 32) * 1024 <= 16384
    big = replace(cfg, ncx=200, ncy=200)
    a = _run(hm, small, st, bonds, True, blocks)
    led = _same(a, _run(hm, big, st, bonds, True, blocks), bonds is not None)
    assert led["status"] == 0 and (led["rebuilds"] >= 2 or side < 22)


def test_indenter_without_bonds(hm):
    """An engine with an indenter but no bond slots takes the bonded build with none."""
    from dataclasses import replace
    cfg, st = dense_gas(30, seed=5, precision=32, sigma_v=0.01)
    top = int(np.argmax(st["pos"][:, 1] + st["radius"]))   # the indenter starts on the highest disc
    x, y = st["pos"][top]
    cfg = replace(cfg, indenter_center=(float(x), float(y + st["radius"][top] + 2e-3 - 1e-7)),
                  indenter_velocity=(0.0, -0.5), indenter_radius=2e-3, load_capacity=64)
    a = _run(hm, cfg, st, None, True, (50,))
    b = _run(hm, cfg, st, None, False, (50,))
    assert np.array_equal(a.load_curve(), b.load_curve()) and np.abs(a.load_curve()).max() > 0.0
    _same(a, b, False)


def test_grid_barrier_wait_runs_out_and_the_engine_recovers(hm):
    """A barrier that may not wait gives up in every block but the last to arrive: the step
    raises, and after a normal budget and a fresh state the engine steps as a fresh one."""
    from tensordem_gb300 import _lib
    cfg, st = dense_gas(64, seed=41, precision=32)
    a = _run(hm, cfg, st, None, True, (3,))
    assert _lib.lib().tdem_hm_set_wait_budget(a._h, 0) == 0
    with pytest.raises(RuntimeError, match="bounded wait"):
        a.step(5)
    assert a.ledger()["status"] & 16
    assert _lib.lib().tdem_hm_set_wait_budget(a._h, 2_000_000_000) == 0
    a.set_state(st["pos"], st["vel"], st["omega"], st["radius"], st["mass"], st["inertia"])
    a.step(20)
    b = _run(hm, cfg, st, None, True, (20,))
    _same(a, b, False)
