"""Eight lanes per atom in the CV passes of small systems (STEINH L, STEINH Q,
STRU_FACTOR) against the FP64 oracle: atom counts at the edges of the 32-atom
blocks, one and two orders, smooth and step pair switches, smooth CV switches,
atoms out of the group, the virial, and the caller-order force pass on pinned
host memory; and STEINH L, Q and Debye on both sides of the rule.

Tolerances of the parity tests: FP64 1e-9 (CV) and 1e-8 (forces), mixed 2e-5
and 2e-3 of the largest force component.
"""
import numpy as np
import pytest

import helpers as H
import mtd
import oracle as O
import systems

pytestmark = pytest.mark.gpu
TOL = {"fp64": (1e-9, 1e-8), "mixed": (2e-5, 2e-3)}


def _cut(n, seed):
    """n atoms of a jittered FCC block that fills the box, the rest left out."""
    nc = max(4, int(np.ceil((n / 4) ** (1 / 3))))
    L = np.array([nc * 5.26] * 3)
    return np.ascontiguousarray(systems.wrap(systems.jitter(systems.fcc(nc, 5.26)[:n], 0.15, seed), L)), L


@pytest.mark.parametrize("n", [1, 31, 33, 500, 2047])
@pytest.mark.parametrize("ls,sw,cvsw", [((6,), "STEP", None), ((4, 6), "STEP", None), ((4, 6), "FERMI", None),
                                        ((3,), "FERMI", (0.3, 20.0)), ((4,), "STEP", (0.3, 20.0))])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_steinh_l(n, ls, sw, cvsw, precision):
    x, L = _cut(n, n + 1)
    a = ["GAUSSIAN", 0.01, 0.005, 9.0, "PACE", 1, "CAL", "NAME", "SWR", "SW_FUNC", sw, "r_0", 3.9]
    a += ["alpha", -8.0] if sw == "FERMI" else []
    if cvsw:
        a += ["CAL", "NAME", "SWC", "SW_FUNC", "FERMI", "r_0", cvsw[0], "alpha", cvsw[1]]
    for l in ls:
        a += ["CAL", "NAME", "Q%d" % l, "STEINH", "L", l, "g", "cutoff_r", 3.9, "SW_FUNC_r", "SWR"]
    for d, l in enumerate(ls):
        a += ["SYMBOL", "v%d" % (d + 1), "Q%d.MEAN_SOLID%s" % (l, ".SWC" if cvsw else "")]
    a += ["CV_dim", len(ls)]
    for d in range(len(ls)):
        a += ["DIM", d + 1, 0.0, 1.0, 100, "v%d" % (d + 1)]
    a += ["WT", 0]
    mask = np.where(np.random.default_rng(n).random(n) < 0.85, 3, 1).astype(np.int32)
    mask[0] = 3
    sel = (mask & 2) != 0
    swr = O.make_sw("STEP", r0=3.9) if sw == "STEP" else O.make_sw("FERMI", r0=3.9, alpha=-8.0)
    rc = 3.9 if sw == "STEP" else 3.9 + np.log(1e6 - 1) / 8.0
    swc = O.make_sw("FERMI", r0=cvsw[0], alpha=cvsw[1]) if cvsw else None
    o = [O.steinh_l(l, x, L, rc, swr, 1e-6, swc, "MEAN_SOLID", ingroup=sel.astype(np.int32)) for l in ls]
    g = O.Grid([[0, 1]] * len(ls), [100] * len(ls), 0.01, 0.005, 9.0, 300.0, 8.617343e-5, False)
    s = [v["cv"] for v in o]
    g.add_hill(s)
    _, dV = g.value(s)
    fo = -sum(dV[d] * o[d]["grad"] for d in range(len(ls)))
    import torch
    f_pinned = torch.zeros((n, 3), dtype=torch.float64).pin_memory().numpy()
    for virial, f in ((True, np.zeros_like(x)), (False, f_pinned)):
        m = mtd.Metad(a, precision=precision, groups={"all": 1, "g": 2})
        m.set_box([0, 0, 0], L)
        v = m.post_force(0, x, f, mask=mask, virial=virial)
        for d in range(len(ls)):
            assert abs(m.cv[d] - s[d]) <= TOL[precision][0] * max(abs(s[d]), 1e-3)
        assert np.abs(f - fo).max() <= TOL[precision][1] * max(np.abs(fo).max(), 1e-12)
        if virial:
            vo = np.array([(f[:, p] * x[:, q]).sum() for p, q in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))])
            assert np.allclose(v, vo, rtol=1e-10, atol=1e-12 * np.abs(f * x).sum() + 1e-300)
        m.close()


@pytest.mark.parametrize("n", [33, 16384, 16385, 32768, 32769])
@pytest.mark.parametrize("kind", ["Q", "SF", "L"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_both_sides_of_the_rule(n, kind, precision):
    x, L = _cut(n, n)
    a = ["GAUSSIAN", 0.01, 0.005, 9.0, "PACE", 1]
    if kind == "Q":
        a += ["CAL", "NAME", "C", "STEINH", "Q", 6, "all", "cutoff_r", 3.9, "cutoff_Natoms", 10, "SYMBOL", "v1", "C.AVE"]
        o = O.steinh_q(6, x, L, 3.9, 10, grad=True)
    elif kind == "SF":
        a += ["CAL", "NAME", "C", "STRU_FACTOR", "all", "cutoff_r", 6.0, "q_factor", 2.8, "SYMBOL", "v1", "C.AVE"]
        o = O.debye(x, L, 6.0, 2.8)
    else:
        a += ["CAL", "NAME", "S", "SW_FUNC", "STEP", "r_0", 3.9, "CAL", "NAME", "C", "STEINH", "L", 6, "all",
              "cutoff_r", 3.9, "SW_FUNC_r", "S", "SYMBOL", "v1", "C.MEAN_SOLID"]
        o = H.oracle_local(x, L, 6)
    a += ["CV_dim", 1, "DIM", 1, 0.0, 2.0, 400, "v1", "WT", 0]
    m = mtd.Metad(a, precision=precision)
    m.set_box([0, 0, 0], L)
    f = np.zeros_like(x)
    m.post_force(0, x, f)
    g = O.Grid([[0.0, 2.0]], [400], 0.01, 0.005, 9.0, 300.0, 8.617343e-5, False)
    g.add_hill([o["cv"]])
    _, dV = g.value([o["cv"]])
    fo = -dV[0] * o["grad"]
    assert H.rel(m.cv[0], o["cv"]) < TOL[precision][0]
    assert np.abs(f - fo).max() <= TOL[precision][1] * np.abs(fo).max()
    m.close()
