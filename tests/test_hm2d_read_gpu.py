"""The one-pass state read-back at odd counts: device tensors, host arrays and device arrays that
are aligned to 8 bytes only must hold the same values, in FP32, FP64 and the FP64-sum form, with
and without bonds, before the first step and later.
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


@pytest.mark.parametrize("case,precision,sums", [((3,), 32, 32), ((17,), 32, 32), ((17,), 64, 32), ((33,), 32, 64),
                                                 ((15, 7), 32, 32), ((15, 7), 64, 32)])
def test_every_destination_holds_the_same_state(hm, case, precision, sums):
    from dataclasses import replace

    from tensordem_gb300 import _lib
    if len(case) == 1:
        cfg, st = dense_gas(case[0], seed=5, precision=precision)
        bonds = None
    else:
        cfg, st, *bonds = small_sheet(*case, precision=precision, speed=20.0)
    cfg = replace(cfg, sum_precision=sums)
    n = cfg.n
    assert n % 2 == 1
    e = hm.HM2D(cfg)
    e.set_state(st["pos"], st["vel"], st["omega"], st["radius"], st["mass"], st["inertia"])
    if bonds is not None:
        e.set_bonds(*bonds)
    for steps in (0, 40):
        e.step(steps)
        got = {k: t.cpu().numpy() for k, t in e.state().items()}
        pos, vel, omega = np.empty((n, 2)), np.empty((n, 2)), np.empty(n)
        e.read_state_host(pos, vel, omega)
        for name, a in (("pos", pos), ("vel", vel), ("omega", omega)):
            assert np.array_equal(got[name], a), name
        flat = {k: torch.full((2 * n + 1,), float("nan"), dtype=torch.float64, device="cuda") for k in got}
        rc = _lib.lib().tdem_hm_read_state(e._h, *[flat[k].data_ptr() + 8 for k in
                                                   ("pos", "vel", "omega", "force", "torque")], 0,
                                           torch.cuda.current_stream().cuda_stream)
        assert rc == 0
        for name, a in got.items():
            assert np.array_equal(flat[name][1:1 + a.size].cpu().numpy(), a.ravel()), name
            assert torch.isnan(flat[name][0])
