"""The 3-D ledger under the lane mappings, entry by entry, against one thread a particle.

Both sum the same terms (the states are the same bits) per thread of another shape, so an entry may
differ by the rounding of its sum: n terms of one sign by n eps relative, terms of either sign by n eps
of the sum of their magnitudes. Counts and the smallest break margin do not depend on the order.
"""

import numpy as np
import pytest
import torch

from tests.test_icedem3d_mappings_gpu import _run

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps
REACTION, PLATENS, FRICTION, ROLLING, CONTACT, COUNTS, MARGIN = slice(0, 3), slice(3, 9), 9, 10, 11, slice(12, 16), 16


@pytest.mark.parametrize("size,squeeze,kw", [
    ((5, 3, 2), True, dict(friction_coefficient=0.3, rolling_resistance_coefficient=0.1)),
    ((9, 7, 5), True, dict(friction_coefficient=0.3, contact_model="hertz")),
    ((20, 15, 8), False, dict(friction_coefficient=0.3)),
    ((17, 16, 9), False, dict(friction_coefficient=0.3, rolling_resistance_coefficient=0.1)),
])
def test_entries_agree(size, squeeze, kw):
    if not torch.cuda.is_available():
        pytest.fail("CUDA GPU required for -m gpu tests")
    a, b = _run("lanes", size, squeeze, 7, **kw), _run("particle", size, squeeze, 7, **kw)
    la, lb = a.read_ledger(), b.read_ledger()
    n = lb[12]
    assert n > 0 and lb[14] == 40 and lb[MARGIN] < 1.0
    assert np.array_equal(la[COUNTS], lb[COUNTS]) and la[MARGIN] == lb[MARGIN]
    assert np.array_equal(la[PLATENS], lb[PLATENS])   # no platens: zeros
    for q in (CONTACT, ROLLING):
        assert abs(la[q] - lb[q]) <= n * EPS * abs(lb[q])
    assert lb[CONTACT] > 0.0 and (lb[ROLLING] != 0.0) == ("rolling_resistance_coefficient" in kw)
    # friction: |F_t . v| of a pair is at most mu F_n |v|; a pair's normal force at most the largest force
    # on a particle of the last evaluation, its relative speed twice the largest speed
    particles = len(b.positions)
    speed = 2.0 * float(b.velocities.norm(dim=1).max())
    force = float(b.forces()[0].norm(dim=1).max()) + 1e-3 * b.config.contact_stiffness * b.config.radius
    assert lb[FRICTION] != 0.0
    assert abs(la[FRICTION] - lb[FRICTION]) <= n * EPS * n * 0.3 * force * speed
    assert np.abs(la[REACTION] - lb[REACTION]).max() <= particles * EPS * max(np.abs(lb[REACTION]).max(), 1e-300)
