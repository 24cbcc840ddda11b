"""One context stepped through its host and its device entry points in turn, and
through errors and replays in between.  STEINH Q splits an atom's neighbours over
eight lanes up to 16,384 atoms (STRU_FACTOR up to 28,672, in FP64 22,528), from host
arrays up to 32,768, and the bias kernel has to read the partial sums of the split
that ran.

Tolerance against the oracle: FP64 sums of n atoms in another order, 1e-12
relative; forces 1e-10 of the largest.
"""
import numpy as np
import pytest

import mtd
import oracle as O

pytestmark = pytest.mark.gpu

RC, CAP = 4.0, 7


def _args(kind="Q"):
    cal = ["STEINH", "Q", 4, "all", "cutoff_r", RC, "cutoff_Natoms", CAP] if kind == "Q" else \
        ["STRU_FACTOR", "all", "cutoff_r", RC, "q_factor", 2.8]
    return ["GAUSSIAN", 0.01, 0.005, 10.0, "PACE", 1, "CAL", "NAME", "C"] + cal + \
        ["SYMBOL", "v1", "C.AVE", "CV_dim", 1, "DIM", 1, 0.0, 1.0, 400, "v1", "WT", 0]


def _system(n):
    L = np.array([(n / 0.03) ** (1 / 3)] * 3)
    return np.ascontiguousarray(np.random.default_rng(n).random((n, 3)) * L), L


def _device(m, step, x):
    import torch

    d_x, d_f = torch.from_numpy(x).cuda(), torch.zeros(x.shape, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    m.post_force_device(step, len(x), d_x.data_ptr(), d_f.data_ptr(), d_f.data_ptr())
    m.sync()
    return m.cv.copy(), d_f.cpu().numpy()


def _host(m, step, x):
    f = np.zeros_like(x)
    m.post_force(step, x, f)
    return m.cv.copy(), f


@pytest.mark.parametrize("kind,n", [("Q", 16384), ("Q", 16385), ("Q", 20000), ("Q", 32768), ("Q", 32769),
                                    ("SF", 22528), ("SF", 22529), ("SF", 28673), ("SF", 32769)])
def test_host_and_device_steps_in_turn(kind, n):
    x, L = _system(n)
    o = O.steinh_q(4, x, L, RC, CAP) if kind == "Q" else O.debye(x, L, RC, 2.8)
    m = mtd.Metad(_args(kind), precision="fp64")
    m.set_box([0, 0, 0], L)
    for step, call in enumerate((_device, _host, _host, _device, _device, _host)):
        cv, f = call(m, step, x)
        assert abs(cv[0] - o["cv"]) <= 1e-12
        s = (f * o["grad"]).sum() / (o["grad"] ** 2).sum()     # the slope the grid gives at this step
        assert np.abs(f - s * o["grad"]).max() <= 1e-10 * np.abs(s * o["grad"]).max()
    m.close()


@pytest.mark.parametrize("call", [_host, _device])
@pytest.mark.parametrize("n", [5000, 20000])
def test_a_replay_after_a_refused_step_leaves_the_right_plan(call, n, tmp_path):
    x, L = _system(n)
    o = O.steinh_q(4, x, L, RC, CAP)
    hills = tmp_path / "HILLS"
    hills.write_text("0 0.3 0.005 0.01\n")
    m = mtd.Metad(_args(), precision="fp64")
    with pytest.raises(mtd.MetadError, match="mtd_set_box"):
        call(m, 0, x)
    m.hills_replay(str(hills))
    m.set_box([0, 0, 0], L)
    cv, _ = call(m, 0, x)
    assert abs(cv[0] - o["cv"]) <= 1e-12
    m.close()
