"""A wait that ran out is named: a grid barrier of the resident steps, a bulk copy of variants 4 to 6."""

import pytest
import torch

from tests._hm_cases import dense_gas

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant,what", [(0, "grid barrier"), (10, "grid barrier"), (4, "bulk copy")])
def test_the_message_names_the_wait(variant, what):
    if not torch.cuda.is_available():
        pytest.fail("CUDA GPU required for -m gpu tests")
    from tensordem_gb300 import _lib, hm2d
    cfg, st = dense_gas(64, seed=41, precision=32)
    e = hm2d.HM2D(cfg)
    e.variant = variant
    e.set_state(st["pos"], st["vel"], st["omega"], st["radius"], st["mass"], st["inertia"])
    e.step(3)
    assert _lib.lib().tdem_hm_set_wait_budget(e._h, 0) == 0
    with pytest.raises(RuntimeError, match=f"bounded wait on a {what}"):
        e.step(5)
