"""Batched network kernels at the sizes where their work is split differently:
one 128-point tile per block (up to 148 tiles) or per warpgroup, partial and
whole tiles, blocks with several tiles, one to four inputs; and the training
gradient of partial tiles.

Tolerances as in tests/test_gpu_nnbias.py (the device uses the SFU exp; a BF16
rounding can flip by one unit): V within 2e-3 of max |V|, dV/ds within 5e-3 of
its largest component, each gradient block within 2e-2 of its largest entry.
"""
import numpy as np
import pytest

import mlp_oracle as MO
import mtd
import systems
from test_gpu_nnbias import _block_rel, _random_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npts,D", [(127, 4), (128, 3), (129, 1), (148 * 128, 4), (148 * 128 + 1, 2),
                                    (4 * 148 * 128 + 5, 4)])
def test_device_batch_matches_oracle(npts, D):
    import torch

    w = _random_params(npts % 97)
    lo, hi = systems.CV4_LO[:D], systems.CV4_HI[:D]
    nb = mtd.NNBias(lo, hi)
    nb.set_params(w, 0.7)
    p = lo + (hi - lo) * np.random.default_rng(npts).random((npts, D))
    u = MO.normalise(p, lo, hi)
    y, gu = MO.input_grad(w, u)
    Vo, dVo = 0.7 * y, 0.7 * gu[:, :D] * 2.0 / (hi - lo)
    d_p = torch.from_numpy(p).cuda()
    d_v = torch.full((2, npts), np.nan, dtype=torch.float64, device="cuda")
    d_g = torch.full((npts, D), np.nan, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    nb.eval_device(npts, d_p.data_ptr(), d_v[0].data_ptr(), d_g.data_ptr(), use_nn=1)
    nb.eval_device(npts, d_p.data_ptr(), d_v[1].data_ptr(), 0, use_nn=1)
    nb.sync_device()
    torch.cuda.synchronize()
    V = d_v.cpu().numpy()
    assert np.abs(V[0] - Vo).max() <= 2e-3 * np.abs(Vo).max()
    assert np.abs(d_g.cpu().numpy() - dVo).max() <= 5e-3 * np.abs(dVo).max()
    assert np.array_equal(V[0], V[1])
    hV, hG = nb.eval(p)
    assert np.abs(hV - Vo).max() <= 2e-3 * np.abs(Vo).max()
    assert np.abs(hG - dVo).max() <= 5e-3 * np.abs(dVo).max()
    nb.close()


@pytest.mark.parametrize("npts", [1, 127, 129, 1300])
def test_training_gradient_of_partial_tiles(npts):
    w = _random_params(12)
    nb = mtd.NNBias(systems.CV4_LO, systems.CV4_HI)
    nb.set_params(w, 1.0)
    p = systems.CV4_LO + (systems.CV4_HI - systems.CV4_LO) * np.random.default_rng(npts).random((npts, 4))
    t = np.sin(3 * p[:, 0]) * np.cos(2 * p[:, 1]) + p[:, 2] * p[:, 3]
    g, loss = nb.loss_grad(p, t, 1.0)
    go, lo = MO.loss_grad(w, MO.normalise(p, systems.CV4_LO, systems.CV4_HI), t)
    assert abs(loss - lo) <= 1e-3 * lo
    for a, b in [(MO.O_W1, MO.O_B1), (MO.O_B1, MO.O_W2), (MO.O_W2, MO.O_B2), (MO.O_B2, MO.O_W3),
                 (MO.O_W3, MO.O_B3), (MO.O_B3, MO.NP)]:
        assert _block_rel(g, go, a, b) < 2e-2, (a, b, _block_rel(g, go, a, b))
    nb.close()


@pytest.mark.parametrize("D,npts", [(4, 2048), (4, 4097), (3, 9001)])
def test_training_gradient_of_points_in_pieces(D, npts):
    # the points cross in pieces of 8,192 doubles; the loss is a sum over all of
    # them (1e-6: FP32 tile sums of equal terms, added in FP64), whatever the call before left
    w = _random_params(13)
    nb = mtd.NNBias(systems.CV4_LO[:D], systems.CV4_HI[:D])
    nb.set_params(w, 1.0)
    rng = np.random.default_rng(npts)
    p = systems.CV4_LO[:D] + (systems.CV4_HI - systems.CV4_LO)[:D] * rng.random((npts, D))
    t = np.sin(3 * p[:, 0]) + p[:, 1] * p[:, -1]
    nb.loss_grad(p[::-1].copy(), t, 1.0)
    g, loss = nb.loss_grad(p, t, 1.0)
    part = [nb.loss_grad(p[a:a + 128], t[a:a + 128], 1.0) for a in range(0, npts, 128)]
    n = [len(p[a:a + 128]) for a in range(0, npts, 128)]
    lo = sum(k * l for k, (_, l) in zip(n, part)) / npts
    assert abs(loss - lo) <= 1e-6 * lo
    go = sum(k * x.astype(np.float64) for k, (x, _) in zip(n, part)) / npts
    assert np.abs(g - go).max() <= 2e-2 * np.abs(go).max()
    nb.close()
