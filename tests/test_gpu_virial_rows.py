"""The virial sums one row per block of each unit's force pass.  A context stepped
with many atoms and then with few keeps the rows of the larger step behind the
smaller one's, and each unit of a deck has its own number of rows: the virial has
to be the sum over r (x) delta f of the step's own forces.

Tolerance: FP64 sums of n products, 1e-12 of the sum of their magnitudes.
"""
import numpy as np
import pytest

import mtd

pytestmark = pytest.mark.gpu

CALS = {
    "SK": ["STRU_FACTOR_K", "all", "nk", 5, "kmag", 2.0, "seed", 3],
    "SF": ["STRU_FACTOR", "all", "cutoff_r", 4.0, "q_factor", 2.8],
    "Q": ["STEINH", "Q", 4, "all", "cutoff_r", 4.0, "cutoff_Natoms", 7],
    "L": ["STEINH", "L", 6, "all", "cutoff_r", 4.0, "SW_FUNC_r", "SW"],
}


def _args(kinds):
    a = ["GAUSSIAN", 0.05, 0.005, 10.0, "PACE", 1, "CAL", "NAME", "SW", "SW_FUNC", "STEP", "r_0", 4.0]
    for k in kinds:
        a += ["CAL", "NAME", "C" + k] + CALS[k]
    for i, k in enumerate(kinds):
        a += ["SYMBOL", "v%d" % (i + 1), "C%s.%s" % (k, "MEAN_SOLID" if k == "L" else "AVE")]
    a += ["CV_dim", len(kinds)]
    for i in range(len(kinds)):
        a += ["DIM", i + 1, -1.0, 3.0, 40, "v%d" % (i + 1)]
    return a + ["WT", 0]


@pytest.mark.parametrize("kinds", [("SK",), ("SK", "SF"), ("L", "SK"), ("Q", "SK", "L"), ("SF", "Q")])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_virial_after_a_larger_step(kinds, precision):
    rng = np.random.default_rng(len(kinds))
    m = mtd.Metad(_args(kinds), precision=precision)
    for step, n in enumerate((20000, 16000, 1000, 33, 5000, 16385, 300)):
        L = np.array([max(14.0, (n / 0.03) ** (1 / 3))] * 3)
        m.set_box([0, 0, 0], L)
        x = np.ascontiguousarray(rng.random((n, 3)) * L)
        f = np.zeros_like(x)
        v = m.post_force(step, x, f, virial=True)
        for t, (a, b) in enumerate(((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))):
            assert abs(v[t] - (f[:, a] * x[:, b]).sum()) <= 1e-12 * np.abs(f[:, a] * x[:, b]).sum() + 1e-18
    m.close()
