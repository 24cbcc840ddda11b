"""Neighbour sets of rational pair switches whose FP32 value says nothing about
the FP64 criterion: next to the pole that an odd power has below d0, and next to
the 0/0 point of the general n / m form.  Isolated pairs, their distances within
1e-6 of that point; the set has to be that of r <= bound and f(r) >= eps in FP64.
"""
import numpy as np
import pytest

import mtd

pytestmark = pytest.mark.gpu

EPS = 0.1


def _pairs(at, seed):
    rng = np.random.default_rng(seed)
    side = 6
    L = np.array([20.0 * side] * 3)
    c = 10.0 + 20.0 * np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)
    c = c + rng.uniform(-1, 1, c.shape)
    u = rng.normal(size=c.shape)
    u /= np.linalg.norm(u, axis=1)[:, None]
    return np.ascontiguousarray(np.concatenate([c, c + (at + rng.uniform(-1e-6, 1e-6, len(c)))[:, None] * u])), L


def _f(r, d0, r0, n, m):
    y = (r - d0) / r0
    with np.errstate(divide="ignore", invalid="ignore"):
        return 1 / (1 + y ** n) if 2 * n == m else (1 - y ** n) / (1 - y ** m)


@pytest.mark.parametrize("d0,r0,n,m,at", [(5.0, 1.0, 3, 6, 4.0), (5.0, 1.0, 5, 10, 4.0), (2.5, 1.7, 8, 20, 4.2)])
@pytest.mark.parametrize("variant", [0, 1])
@pytest.mark.parametrize("skin", [False, True])
def test_the_set_is_the_fp64_criterions(d0, r0, n, m, at, variant, skin):
    a = ["GAUSSIAN", 0.01, 0.005, 10.0, "PACE", 1, "CAL", "NAME", "SW", "SW_FUNC", "RATIONAL", "r_0", r0, "d_0", d0,
         "n", n, "m", m, "CAL", "NAME", "C", "STEINH", "L", 6, "all", "cutoff_eps", EPS, "SW_FUNC_r", "SW",
         "SYMBOL", "v1", "C.MEAN_SOLID", "CV_dim", 1, "DIM", 1, 0.0, 2.0, 400, "v1", "WT", 0]
    if skin:
        a += ["NEIGH_SKIN", 0.5, "NEIGH_EVERY", 10]
    x, L = _pairs(at, n)
    h = len(x) // 2
    d = x[h:] - x[:h]
    r = np.sqrt(d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2])
    want = (_f(r, d0, r0, n, m) >= EPS).astype(np.int32)
    M = mtd.Metad(a, precision="mixed")
    M.set_box([0, 0, 0], L)
    M.set_tuning(variant, 0, 0)
    f = np.zeros_like(x)
    try:
        M.post_force(0, x, f)
    except mtd.MetadError as e:   # a force next to a pole is no finite number: the lists stand
        assert mtd.STATUS_NAMES.get(e.status) == "NAN"
    count, _ = M.neighbors("C", len(x))
    assert np.array_equal(count, np.concatenate([want, want]))
    M.close()
