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


@pytest.mark.parametrize("n", [100, 5000, 108000, 250000])
@pytest.mark.parametrize("nk", [3, 24])
def test_mixed_terms_join_an_fp64_sum(n, nk):
    """n atoms at one place: every term is the same FP32 number, its n-fold sum is
    exact in FP64, so S(k) is n times that of one atom up to FP64 roundings (a few
    2^-53 of the squares, their sums over k, the mean)."""
    at = np.array([[11.3, 4.7, 29.9]])
    one, _, _ = _step(at, nk, "mixed", L=[64.0] * 3)
    cv, _, _ = _step(np.tile(at, (n, 1)), nk, "mixed", L=[64.0] * 3, hi=4.0 * n)
    assert abs(cv - n * one) <= n * (nk + 8) * 2.0 ** -52


@pytest.mark.parametrize("nk,far", [(13, 0), (129, 40)])
@pytest.mark.parametrize("virial", [False, True])
def test_mixed_forces_do_not_depend_on_the_atoms_per_thread(nk, far, virial):
    """The same group of 20,000 atoms alone (one atom a thread in the force pass) and
    with 160,000 others outside the group (two), some of the group so far out that
    their phases leave the base's range: the FP32 sums over k are the same, and the
    forces with them up to the FP64 sum over atoms, taken over other blocks
    (1e-16 of it each, 2^-44 allowed; an FP32 sum in another order differs by 2^-24)."""
    rng = np.random.default_rng(nk)
    L = np.array([150.0] * 3)
    x = rng.random((180000, 3)) * L
    x[rng.choice(20000, far, replace=False)] += L * rng.integers(9000, 12000, (far, 3))
    mask = np.where(np.arange(len(x)) < 20000, 3, 1).astype(np.int32)
    cv1, f1, _ = _step(x[:20000].copy(), nk, "mixed", L=L, mask=mask[:20000], virial=virial)
    cv2, f2, _ = _step(x, nk, "mixed", L=L, mask=mask, virial=virial)
    assert abs(cv1 - cv2) <= 1e-13 * cv1 and not np.any(f2[20000:])
    assert np.abs(f1).max() > 0 and np.all(np.abs(f1 - f2[:20000]) <= 2.0 ** -44 * np.abs(f1))
