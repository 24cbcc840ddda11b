"""The network far outside the box: hidden units driven to -200 and to -1e33 are
both exactly off (a SiLU and its derivative vanish where exp(-z) overflows), so
the values and gradients there are the same, and those of the output biases."""
import numpy as np
import pytest

import mlp_oracle as MO
import mtd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npts", [3, 128 * 150])
def test_units_far_below_zero_are_off(npts):
    import torch

    rng = np.random.default_rng(3)
    w = np.zeros(MO.NP, dtype=np.float32)
    w[MO.O_W1:MO.O_B1].reshape(MO.H, MO.IN)[:, 0] = -1.0
    w[MO.O_W2:MO.O_B2] = rng.normal(0, np.sqrt(2 / MO.H), MO.H * MO.H)
    w[MO.O_B2:MO.O_W3] = rng.normal(0, 0.1, MO.H)
    w[MO.O_W3:MO.O_B3] = rng.normal(0, np.sqrt(1 / MO.H), MO.H)
    nb = mtd.NNBias(np.zeros(4), np.ones(4))
    nb.set_params(w, 1.0)
    p = np.full((npts, 4), 0.5)
    u = np.where(np.arange(npts) % 3 == 0, 200.0, np.where(np.arange(npts) % 3 == 1, 1e33, 3e36))
    p[:, 0] = 0.5 * (u + 1)
    d_p = torch.from_numpy(p).cuda()
    d_v = torch.zeros(npts, dtype=torch.float64, device="cuda")
    d_g = torch.zeros((npts, 4), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    nb.eval_device(npts, d_p.data_ptr(), d_v.data_ptr(), d_g.data_ptr(), use_nn=1)
    nb.sync_device()
    torch.cuda.synchronize()
    V = d_v.cpu().numpy()
    b2 = w[MO.O_B2:MO.O_W3].astype(np.float64)
    bf = torch.from_numpy(w[MO.O_W3:MO.O_B3]).bfloat16().double().numpy()
    want = (bf * b2 / (1 + np.exp(-b2))).sum()
    assert np.all(V == V[0]) and abs(V[0] - want) <= 128 * 2.0 ** -22 * np.abs(bf * b2).max()
    assert not np.any(d_g.cpu().numpy())
    nb.close()
