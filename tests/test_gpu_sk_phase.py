"""S(k): the phases taken from the low word of a based FP64 sum
(csrc/common.cuh, kTurnBase) and the pairs of k-vectors.

Odd and even k counts at the edges of the 64-pair tiles, atom counts at the
edges of the 256-atom blocks and 512-atom chunks, groups, and positions so far
out that the phase leaves the base's range (|u| >= 2^18 half turns), which take
the FP64 rounding instead.

Tolerance: an FP32 sin or cos is within 2e-7 of the exact one (its evaluation
error; the based phase adds 1.6e-9), so rho is within N * 2e-7 * sqrt(2) of the
FP64 sum, S(k) = |rho|^2 / N within 2 |rho| / N of that, and a force component
within 2 a / N of sum_k |k| (2e-7 sqrt(2) |rho| + the error of rho), with FP32
sums over k (K 2^-24 relative).  Phases carry the FP64 rounding of u
itself, a few |u| 2^-53.  In FP64 mode the same with 4e-16 for the sine's error.
"""
import numpy as np
import pytest

import mtd
import oracle as O
import systems

pytestmark = pytest.mark.gpu


def _args(nk, group="all"):
    return ["GAUSSIAN", 0.5, 0.005, 10.0, "PACE", 10,
            "CAL", "NAME", "SK", "STRU_FACTOR_K", group, "nk", nk, "kmag", systems.KMAG_111, "seed", 9,
            "SYMBOL", "v1", "SK.AVE", "CV_dim", 1, "DIM", 1, 0.0, 100.0, 500, "v1", "WT", 0]


@pytest.mark.parametrize("n,nk,far", [(1, 1, 0), (255, 3, 0), (257, 8, 0), (511, 9, 3), (513, 15, 0), (2049, 17, 40),
                                      (3000, 129, 0), (1025, 300, 1), (76031, 24, 5), (160001, 5, 0)])
@pytest.mark.parametrize("virial", [False, True])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_matches_fp64_sum(n, nk, far, virial, precision):
    nc = int(np.ceil((n / 4) ** (1 / 3)))
    L = np.array([nc * 5.26] * 3)
    x = systems.wrap(systems.jitter(systems.fcc(nc, 5.26)[:n], 0.2, n), L)
    rng = np.random.default_rng(n)
    if far:   # whole box lengths away, up to 3e6 half turns
        x[rng.choice(n, far, replace=False)] += L * rng.integers(200000 // nc, 300000 // nc, (far, 3))
    x = np.ascontiguousarray(x)
    mask = np.where(rng.random(n) < 0.8, 3, 1).astype(np.int32)
    mask[0] = 3
    m = mtd.Metad(_args(nk, "g"), precision=precision, groups={"all": 1, "g": 2})
    m.set_box([0, 0, 0], L)
    f = np.zeros_like(x)
    v = m.post_force(0, x, f, mask=mask, virial=virial)
    k = systems.kvectors(nk, systems.KMAG_111, 9)
    sel = (mask & 2) != 0
    N = sel.sum()
    ph = x[sel] @ k.T
    rho = np.exp(1j * ph).sum(0)
    e = (3e-7 if precision == "mixed" else 4e-16) + np.abs(ph).max() * 2.0 ** -50
    drho = N * e if N < 100 else N ** 0.5 * 10 * e      # independent errors beyond a few atoms
    drho = drho + N * 2.0 ** -52
    S = (np.abs(rho) ** 2).mean() / N
    tS = (2 * np.abs(rho) * drho + drho ** 2).mean() / N + 1e-12
    assert abs(m.cv[0] - S) <= tS
    g = O.Grid([[0.0, 100.0]], [500], 0.5, 0.005, 10.0, 300.0, 8.617343e-5, False)
    g.add_hill([m.cv[0]])
    dV = g.value([m.cv[0]])[1][0]
    w = 2.0 / (N * nk) * (-rho.real * np.sin(ph) + rho.imag * np.cos(ph))
    fo = np.zeros_like(x)
    fo[sel] = -dV * (w @ k)
    tol = abs(dV) * 2.0 / (N * nk) * (np.abs(k).max(1) * ((e + nk * (2.0 ** -24 if precision == "mixed" else 2.0 ** -52)) * 1.5 * np.abs(rho) + 2 * drho)).sum()
    assert np.abs(f - fo).max() <= tol + 1e-14 * abs(dV)
    assert np.all(f[~sel] == 0)
    if virial:
        vo = np.array([(f[:, a] * x[:, b]).sum() for a, b in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))])
        assert np.allclose(v, vo, rtol=1e-10, atol=1e-12 * np.abs(f * x).sum())
    m.close()


def test_forces_do_not_depend_on_the_virial_or_the_block_layout():
    """The same atoms with and without the virial, and behind enough other
    atoms for two a thread: the same forces bit for bit."""
    L = np.array([30 * 5.26] * 3)
    x = np.ascontiguousarray(systems.wrap(systems.jitter(systems.fcc(30, 5.26), 0.2, 4), L))
    out = []
    for virial in (False, True):
        m = mtd.Metad(_args(13), precision="mixed")
        m.set_box([0, 0, 0], L)
        f = np.zeros_like(x)
        m.post_force(0, x, f, virial=virial)
        out.append((m.cv.copy(), f))
        m.close()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
