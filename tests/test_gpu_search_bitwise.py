"""The shapes of the neighbour search write the same lists in the same order, so a
step's CVs and forces do not depend on the shape in any bit: the warp-per-atom
search (shape 0) against the thread-per-atom ones (1, 2), with caps, smooth
switches and type-free pairs, on both sides of the one-cluster cell list's 16,384
atoms and of the warp shape's limits.
"""
import numpy as np
import pytest

import mtd
from test_gpu_warp_search import _args

pytestmark = pytest.mark.gpu


def _step(kind, x, L, per, variant, precision):
    m = mtd.Metad(_args(kind), precision=precision)
    m.set_box([0, 0, 0], L, per)
    m.set_tuning(variant, 0, 0)
    f = np.zeros_like(x)
    v = m.post_force(0, x, f, virial=True)
    out = (m.cv.copy(), f, v)
    m.close()
    return out


@pytest.mark.parametrize("kind", ["Q", "SF", "STEP", "FERMI"])
@pytest.mark.parametrize("n,per,rho", [(1023, (1, 1, 1), 0.1), (16384, (1, 1, 1), 0.03), (16385, (1, 0, 1), 0.03),
                                       (65536, (1, 1, 1), 0.03), (65537, (1, 1, 1), 0.03)])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_shapes_agree_in_every_bit(kind, n, per, rho, precision):
    side = max(16.0, (n / rho) ** (1 / 3))
    L = np.array([side, side * 1.1, side])
    x = np.ascontiguousarray(np.random.default_rng(n).random((n, 3)) * L)
    ref = _step(kind, x, L, per, 1, precision)
    for variant in (0, 2):
        for a, b in zip(ref, _step(kind, x, L, per, variant, precision)):
            assert np.array_equal(a, b)
