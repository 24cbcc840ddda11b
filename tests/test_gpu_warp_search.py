"""One warp per atom in the neighbour search (with the cap of STEINH Q ranked by
the same kernel) and the one-cluster cell list, against the thread-per-atom
shape on the same positions: the same lists entry by entry, so the same CVs and
forces bit for bit; and against a brute-force count at small sizes.

Atom counts at the edges of the warps' blocks (8 atoms), of the cluster's
threads (1,024 and 65,536 atoms) and of the rule for the warp shape; open and
periodic boxes, sparse ones on both sides of the cluster's 262,144 cells, a dense system with more than 32 neighbours, caps that bind.
"""
import numpy as np
import pytest

import mtd

pytestmark = pytest.mark.gpu


def _args(kind):
    a = ["GAUSSIAN", 0.01, 0.005, 10.0, "PACE", 1]
    if kind == "Q":
        a += ["CAL", "NAME", "C", "STEINH", "Q", 4, "all", "cutoff_r", 4.0, "cutoff_Natoms", 7, "SYMBOL", "v1", "C.AVE"]
    elif kind == "SF":
        a += ["CAL", "NAME", "C", "STRU_FACTOR", "all", "cutoff_r", 4.0, "q_factor", 2.8, "SYMBOL", "v1", "C.AVE"]
    else:
        sw = ["STEP", "r_0", 4.0] if kind == "STEP" else ["FERMI", "r_0", 3.0, "alpha", -8.0]
        a += ["CAL", "NAME", "SW", "SW_FUNC"] + sw + \
             ["CAL", "NAME", "C", "STEINH", "L", 6, "all", "cutoff_r", 4.0, "SW_FUNC_r", "SW", "SYMBOL", "v1",
              "C.MEAN_SOLID"]
    return a + ["CV_dim", 1, "DIM", 1, 0.0, 2.0, 400, "v1", "WT", 0]


def _run(kind, x, L, per, variant, M, precision):
    m = mtd.Metad(_args(kind), precision=precision)
    m.set_box([0, 0, 0], L, per)
    m.set_tuning(variant, 0, 0)
    f = np.zeros_like(x)
    m.post_force(0, x, f)
    out = (m.cv.copy(), f, m.neighbors("C", x.shape[0], M))
    m.close()
    return out


@pytest.mark.parametrize("n,kind,per,rho", [(1, "STEP", (1, 1, 1), 0.02), (7, "Q", (0, 1, 0), 0.02),
                                            (9, "SF", (1, 1, 1), 0.02), (1023, "Q", (1, 1, 1), 0.13),
                                            (1025, "FERMI", (0, 0, 0), 0.05), (1024, "STEP", (1, 0, 1), 0.15),
                                            (1000, "STEP", (1, 1, 1), 1.25e-4), (1000, "STEP", (1, 1, 1), 1.5e-5),
                                            (4000, "Q", (1, 1, 1), 0.03), (65536, "FERMI", (1, 1, 1), 0.03),
                                            (65537, "SF", (1, 1, 1), 0.03), (131073, "Q", (1, 1, 1), 0.03)])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_same_lists_as_a_thread_per_atom(n, kind, per, rho, precision):
    side = max(16.0, (n / rho) ** (1 / 3))
    L = np.array([side, side * 1.1, side * 0.95 if n > 4000 else side])
    x = np.ascontiguousarray(np.random.default_rng(n).random((n, 3)) * L)
    M = 64 if kind == "Q" else 96
    cv0, f0, (c0, l0) = _run(kind, x, L, per, 1, M, precision)
    cv1, f1, (c1, l1) = _run(kind, x, L, per, 0, M, precision)
    assert np.array_equal(c0, c1) and np.array_equal(l0, l1)
    if n <= 1025 and kind in ("STEP", "SF"):
        d = x[None] - x[:, None]
        d -= np.where(np.array(per) > 0, L * np.rint(d / L), 0.0)
        r2 = (d * d).sum(-1) + np.where(np.eye(n) > 0, 1e9, 0.0)
        assert np.array_equal(c1, (r2 < 16.0).sum(1))
    assert np.allclose(cv0, cv1, rtol=1e-12 if precision == "fp64" else 1e-6)
    assert np.abs(f0 - f1).max() <= (1e-11 if precision == "fp64" else 1e-4) * max(np.abs(f0).max(), 1e-30)
