"""S(k): what the sums keep of the phases' and terms' precision."""
import numpy as np
import pytest

import mtd
import systems

pytestmark = pytest.mark.gpu

SEED = 9


def _step(x, nk, precision, L=None, mask=None, hi=100.0, virial=False):
    args = ["GAUSSIAN", 0.5, 0.005, 10.0, "PACE", 10,
            "CAL", "NAME", "SK", "STRU_FACTOR_K", "all" if mask is None else "g", "nk", nk, "kmag", systems.KMAG_111,
            "seed", SEED, "SYMBOL", "v1", "SK.AVE", "CV_dim", 1, "DIM", 1, 0.0, hi, 500, "v1", "WT", 0]
    m = mtd.Metad(args, precision=precision, groups={"all": 1, "g": 2})
    m.set_box([0, 0, 0], [2.0 ** 22] * 3 if L is None else L)
    f = np.zeros_like(x)
    v = m.post_force(0, np.ascontiguousarray(x), f, mask=mask, virial=virial)
    cv = float(m.cv[0])
    m.close()
    return cv, f, v


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("shift", [0, 7, 14, 20])
def test_fp64_phases_carry_no_rounding_of_their_own(axis, shift):
    """Two atoms, at the origin and 2^shift along an axis: k.x is exact in FP64, so
    S(k) = 1 + cos(k.x) with the sine and cosine each within 2^-52 (two units in
    the last place) and a few roundings: |rho| <= 2, S off by less than 2 |rho| *
    2^-52 * sqrt(2) + 4 * 2^-52 < 10 * 2^-52.  Forces: k |rho| sin(arg), |rho| and
    its phase within 2^-51, the sine within 2^-52, nk terms and their sum."""
    nk = 24
    x = np.zeros((2, 3))
    x[1, axis] = 2.0 ** shift
    k = systems.kvectors(nk, systems.KMAG_111, SEED)
    ph = k[:, axis] * 2.0 ** shift
    cv, f, _ = _step(x, nk, "fp64")
    assert abs(cv - (1 + np.cos(ph)).mean()) <= 10 * 2.0 ** -52
    w = (np.sin(ph)[:, None] * k).sum(0)
    slope = f[1] @ w / (w @ w)     # the bias's own, whatever the grid gives
    assert slope != 0.0
    tol = abs(slope) * np.abs(k).sum(0) * 16 * 2.0 ** -52
    assert np.all(np.abs(f[1] - slope * w) <= tol) and np.all(np.abs(f[0] + slope * w) <= tol)


@pytest.mark.parametrize("far", [2.0 ** 46, 1e16, 3e18, 1e300])
@pytest.mark.parametrize("n", [1, 600])
def test_fp64_phases_without_end_stay_sines_and_cosines(far, n):
    """Atoms at one place, however far out: S(k) = n, and no force."""
    x = np.tile([far, -0.5 * far, 0.25], (n, 1))
    cv, f, _ = _step(x, 5, "fp64", hi=1000.0)
    assert abs(cv - n) <= n * 1e-13
    assert np.abs(f).max() <= 1e-10
