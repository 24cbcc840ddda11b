"""Neighbour lists that outgrow their first size, which comes from the box's mean
density: clusters of atoms in an otherwise empty box."""
import numpy as np
import pytest

import mtd

pytestmark = pytest.mark.gpu

RC = 6.0
L = np.array([45.0, 45.0, 45.0])


def _clusters(members, spare, seed):
    """27 balls of `members` atoms all within RC of one another, and `spare`
    atoms per ball out of everyone's reach of a ball."""
    rng = np.random.default_rng(seed)
    centres = 7.5 + 15.0 * np.stack(np.meshgrid(*[np.arange(3)] * 3, indexing="ij"), -1).reshape(-1, 3)
    x = []
    for c in centres:
        d = rng.normal(size=(members, 3))
        d *= (2.5 * rng.random(members) ** (1 / 3) / np.linalg.norm(d, axis=1))[:, None]
        x.append(c + d)
        x.append(c + 7.4 * np.array([1.0, 1.0, 1.0]) + 0.05 * rng.random((spare, 3)) if spare else np.zeros((0, 3)))
    return np.ascontiguousarray(np.concatenate(x) % L)


def _within(x, rc):
    d = x[None] - x[:, None]
    d -= L * np.rint(d / L)
    r2 = (d * d).sum(-1)
    return (r2 <= rc * rc) & ~np.eye(len(x), dtype=bool), r2


def _nearest(near, r2, cap):
    """The cap nearest of each row's neighbours, ascending."""
    return [np.sort(sorted(np.flatnonzero(a), key=lambda j: (b[j], j))[:cap]) for a, b in zip(near, r2)]


def _q(rc=RC, cap=12):
    return ["CAL", "NAME", "Q", "STEINH", "Q", 4, "all", "cutoff_r", rc, "cutoff_Natoms", cap]


def _deck(cals, symbol="Q.AVE"):
    return ["GAUSSIAN", 0.01, 0.005, 10.0, "PACE", 1] + cals + \
        ["SYMBOL", "v1", symbol, "CV_dim", 1, "DIM", 1, -1.0, 2.0, 400, "v1", "WT", 0]


@pytest.mark.parametrize("variant", [0, 1])
@pytest.mark.parametrize("members,more,cap", [(58, 66, 64), (61, 69, 12), (65, 73, 64)])
def test_a_capped_list_grows_to_64_entries_and_no_further(variant, members, more, cap):
    m = mtd.Metad(_deck(_q(cap=cap)), precision="fp64")
    m.set_box([0, 0, 0], L)
    m.set_tuning(variant, 0, 0)
    x = _clusters(members, more - members, 1)
    near, r2 = _within(x, RC)
    assert near.sum(1).max() == members - 1
    f = np.zeros_like(x)
    m.post_force(0, x, f)
    count, idx = m.neighbors("Q", len(x), 64)
    for k, kept in enumerate(_nearest(near, r2, cap)):
        assert np.array_equal(idx[k, :count[k]], kept)
    x = _clusters(more, 0, 2)
    f = np.zeros_like(x)
    with pytest.raises(mtd.MetadError, match="more than 64 atoms"):
        m.post_force(1, x, f)
    m.close()


@pytest.mark.parametrize("skin", [False, True])
def test_another_cals_long_list_is_no_matter_of_the_capped_one(skin):
    # 90 atoms within 6.0 of one another, up to 55 of them within 2.0
    x = _clusters(90, 0, 3)
    args = _deck(_q(2.0) + ["CAL", "NAME", "SF", "STRU_FACTOR", "all", "cutoff_r", RC, "q_factor", 2.8])
    i = args.index("CV_dim")
    args = args[:i] + ["SYMBOL", "v2", "SF.AVE", "CV_dim", 2, "DIM", 1, -1.0, 2.0, 400, "v1", "DIM", 2, -50.0, 50.0,
                       400, "v2", "WT", 0]
    if skin:
        args += ["NEIGH_SKIN", 0.5, "NEIGH_EVERY", 10]
    m = mtd.Metad(args, precision="fp64")
    m.set_box([0, 0, 0], L)
    near, r2 = _within(x, 2.0)
    assert near.sum(1).max() <= 64 < _within(x, RC)[0].sum(1).max()
    f = np.zeros_like(x)
    m.post_force(0, x, f)
    count, idx = m.neighbors("Q", len(x), 64)
    for k, kept in enumerate(_nearest(near, r2, 12)):
        assert np.array_equal(idx[k, :count[k]], kept)
    count, _ = m.neighbors("SF", len(x))
    assert np.array_equal(count, _within(x, RC)[0].sum(1))
    m.close()
