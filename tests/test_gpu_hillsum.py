"""The batched exact hill sum (csrc/hillsum.cu) against its NumPy restatement.

Sizes at the edges of the 32-point warps, the 32-hill groups and the splits of
the hills over warps and clusters; hills along a trajectory and in random
order, of unequal widths; points outside the box and not finite.

Tolerance, per point: the exponent x = r^2 / (2 s^2) <= 40 carries at most 4
roundings (2^-53 relative each), so a term is off by at most 40 * 4 * 2^-53 =
1.8e-14 relative, plus a few 2^-53 of the evaluation and the sum; hills beyond
the cut miss h e^-40 each.  1e-13 of the sum of the terms' magnitudes.
"""
import numpy as np
import pytest

import mtd
import systems

pytestmark = pytest.mark.gpu


def _hills(n, D, seed, walk):
    rng = np.random.default_rng(seed)
    c = systems.cv4_hills(n=n, seed=seed)[0] if walk else \
        systems.CV4_LO + (systems.CV4_HI - systems.CV4_LO) * rng.random((n, 4))
    return np.ascontiguousarray(c[:, :D]), rng.uniform(-0.002, 0.005, n), rng.uniform(0.01, 0.04, n)


def _sum(p, c, h, s):
    V, dV = np.zeros(len(p)), np.zeros_like(p)
    aV, adV = np.zeros(len(p)), np.zeros_like(p)
    for ck, hk, sk in zip(c, h, s):
        d = p - ck
        e = hk * np.exp(-(d * d).sum(1) / (2 * sk * sk))
        g = -e[:, None] * d / (sk * sk)
        V += e
        dV += g
        aV += np.abs(e)
        adV += np.abs(g)
    return V, dV, aV, adV


@pytest.mark.parametrize("npts,nh,D,walk", [(1, 1, 4, True), (31, 32, 1, True), (32, 33, 2, False), (33, 65, 3, True),
                                            (257, 1000, 4, False), (1000, 1023, 4, True), (5000, 31, 3, False),
                                            (3001, 2500, 4, True)])
def test_batch_matches_oracle(npts, nh, D, walk):
    import torch

    lo, hi = systems.CV4_LO[:D], systems.CV4_HI[:D]
    c, h, s = _hills(nh, D, npts, walk)
    p = lo + (hi - lo) * (1.2 * np.random.default_rng(nh).random((npts, D)) - 0.1)
    nb = mtd.NNBias(lo, hi)
    nb.add_hills(c, h, s)
    V, dV, aV, adV = _sum(p, c, h, s)
    cut = nh * np.abs(h).max() * np.exp(-40.0)
    got = [nb.exact(p)]
    d_p = torch.from_numpy(p).cuda()
    d_v = torch.full((npts,), np.nan, dtype=torch.float64, device="cuda")
    d_g = torch.full((npts, D), np.nan, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    nb.eval_device(npts, d_p.data_ptr(), d_v.data_ptr(), d_g.data_ptr(), use_nn=0)
    torch.cuda.synchronize()
    got.append((d_v.cpu().numpy(), d_g.cpu().numpy()))
    for gv, gd in got:
        assert np.all(np.abs(gv - V) <= 1e-13 * aV + cut)
        assert np.all(np.abs(gd - dV) <= 1e-13 * adV + 10 * cut / s.min())
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
    nb.close()


def test_points_and_hills_that_are_not_finite_count_nothing():
    c, h, s = _hills(70, 4, 3, True)
    p = np.array([c[5], c[40], c[5], c[69]]) + 0.001
    p[1, 2], p[2, 0] = np.nan, np.inf
    # and a hill on a point whose 1 / sigma^2 overflows
    c2 = np.insert(c, [10, 50, 60], [[np.nan] * 4, [np.inf, 0, 0, 0], p[0]], axis=0)
    h2, s2 = np.insert(h, [10, 50, 60], 1.0), np.insert(s, [10, 50, 60], [0.02, 0.02, 1e-155])
    out = []
    for args in ((c, h, s), (c2, h2, s2)):
        nb = mtd.NNBias(systems.CV4_LO, systems.CV4_HI)
        nb.add_hills(*args)
        out.append(nb.exact(p))
        nb.close()
    V, dV, aV, adV = _sum(p[[0, 3]], c, h, s)
    for gv, gd in out:
        assert np.all(gv[1:3] == 0) and np.all(gd[1:3] == 0)
        assert np.all(np.abs(gv[[0, 3]] - V) <= 1e-13 * aV + 1e-18)
        assert np.all(np.abs(gd[[0, 3]] - dV) <= 1e-13 * adV + 1e-15)


def test_batch_replays_from_a_captured_graph():
    import torch

    c, h, s = _hills(300, 4, 8, True)
    nb = mtd.NNBias(systems.CV4_LO, systems.CV4_HI)
    nb.add_hills(c, h, s)
    rng = np.random.default_rng(1)
    p = [systems.CV4_LO + (systems.CV4_HI - systems.CV4_LO) * rng.random((500, 4)) for _ in range(2)]
    d_p = torch.from_numpy(p[0]).cuda()
    d_v, d_g = torch.zeros(500, dtype=torch.float64, device="cuda"), torch.zeros((500, 4), dtype=torch.float64,
                                                                                 device="cuda")
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    st = torch.cuda.Stream()
    with torch.cuda.graph(g, stream=st):
        nb.eval_device(500, d_p.data_ptr(), d_v.data_ptr(), d_g.data_ptr(), use_nn=0, stream=st.cuda_stream)
    for q in p:
        d_p.copy_(torch.from_numpy(q))
        g.replay()
        torch.cuda.synchronize()
        V, dV = nb.exact(q)
        assert np.array_equal(d_v.cpu().numpy(), V) and np.array_equal(d_g.cpu().numpy(), dV)
    del g
    nb.close()


def test_two_threads_on_two_streams_share_one_object():
    import threading

    import torch

    c, h, s = _hills(2000, 4, 9, True)
    nb = mtd.NNBias(systems.CV4_LO, systems.CV4_HI)
    nb.add_hills(c, h, s)
    rng = np.random.default_rng(2)
    sizes = [(700, 9000), (8000, 300)]
    pts = [[systems.CV4_LO + (systems.CV4_HI - systems.CV4_LO) * rng.random((n, 4)) for n in ns] for ns in sizes]
    dev = [[torch.from_numpy(p).cuda() for p in ps] for ps in pts]
    out = [[[torch.zeros(n, dtype=torch.float64, device="cuda"), torch.zeros((n, 4), dtype=torch.float64,
                                                                             device="cuda")] for n in ns]
           for ns in sizes]
    streams = [torch.cuda.Stream() for _ in sizes]
    torch.cuda.synchronize()

    def run(w):
        for _ in range(20):
            for n, p, (v, g) in zip(sizes[w], dev[w], out[w]):
                nb.eval_device(n, p.data_ptr(), v.data_ptr(), g.data_ptr(), use_nn=0,
                               stream=streams[w].cuda_stream)

    ts = [threading.Thread(target=run, args=(w,)) for w in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    torch.cuda.synchronize()
    for w in range(2):
        for p, (v, g) in zip(pts[w], out[w]):
            V, dV = nb.exact(p)
            assert np.array_equal(v.cpu().numpy(), V) and np.array_equal(g.cpu().numpy(), dV)
    nb.close()


def test_widths_at_the_ends_of_the_range():
    # a hill wide enough to reach a stand-in coordinate, and one whose exponent's factor overflows
    p = np.array([[0.1, 0.2, 0.3, 0.4], [np.nan, 0.2, 0.3, 0.4], [0.1, -np.inf, 0.3, 0.4], [0.5, 0.5, 0.5, 0.5]])
    nb = mtd.NNBias(systems.CV4_LO, systems.CV4_HI)
    nb.add_hills(np.array([p[0], p[3]]), np.array([0.25, 0.5]), np.array([1e151, 1.2e-154]))
    V, dV = nb.exact(p)
    assert np.array_equal(V, [0.25, 0.0, 0.0, 0.75]) and not np.any(dV[:3])
    want = -0.25 * (p[3] - p[0]) / 1e302
    assert np.all(np.abs(dV[3] - want) <= 1e-13 * np.abs(want))
    nb.close()


@pytest.mark.parametrize("D", [1, 3, 4])
def test_a_hill_counts_to_the_last_bit_of_its_cut(D):
    """Points at r^2 = 80 sigma^2 (1 -+ 1e-9): within the cut the hill's full value,
    40 * 2e-9 of the exponent off e^-40 at most, beyond it nothing."""
    s = np.array([0.55, 1.1, 1.3])
    e = np.array([-1e-9, 1e-9])
    p = np.zeros((6, D))
    p[:, D - 1] = np.sqrt(80 * s[:, None] ** 2 * (1 + e)).ravel()
    for k in range(3):
        nb = mtd.NNBias(np.full(D, -20.0), np.full(D, 20.0))
        nb.add_hills(np.zeros((1, D)), np.array([1e18]), s[k:k + 1])
        V, dV = nb.exact(p[2 * k:2 * k + 2])
        want = 1e18 * np.exp(-40.0 * (1 - 1e-9))
        assert abs(V[0] - want) <= 1e-12 * want and V[1] == 0
        g = -want * p[2 * k, D - 1] / s[k] ** 2
        assert abs(dV[0, D - 1] - g) <= 1e-12 * abs(g) and not np.any(dV[1])
        nb.close()


@pytest.mark.parametrize("npts,nh,D", [(1, 40, 4), (500, 300, 3), (9000, 5000, 4), (40000, 700, 4)])
def test_a_captured_batch_is_one_kernel_node(npts, nh, D):
    """No memory nodes, so the graph can be instantiated twice and nested; the
    sums are those of a call outside a capture, bit for bit."""
    import torch
    from cuda.bindings import runtime as rt

    def ok(r):
        assert r[0] == rt.cudaError_t.cudaSuccess, r[0]
        return r[1:] if len(r) != 2 else r[1]

    lo, hi = systems.CV4_LO[:D], systems.CV4_HI[:D]
    nb = mtd.NNBias(lo, hi)
    nb.add_hills(*_hills(nh, D, npts, True))
    p = lo + (hi - lo) * np.random.default_rng(npts).random((npts, D))
    d_p = torch.from_numpy(p).cuda()
    d_v, d_g = torch.zeros(npts, dtype=torch.float64, device="cuda"), torch.zeros((npts, D), dtype=torch.float64,
                                                                                  device="cuda")
    torch.cuda.synchronize()
    st = ok(rt.cudaStreamCreateWithFlags(rt.cudaStreamNonBlocking))
    ok(rt.cudaStreamBeginCapture(st, rt.cudaStreamCaptureMode.cudaStreamCaptureModeThreadLocal))
    nb.eval_device(npts, d_p.data_ptr(), d_v.data_ptr(), d_g.data_ptr(), use_nn=0, stream=int(st))
    graph = ok(rt.cudaStreamEndCapture(st))
    n = ok(rt.cudaGraphGetNodes(graph, 0))[1]
    nodes = ok(rt.cudaGraphGetNodes(graph, n))[0]
    assert [ok(rt.cudaGraphNodeGetType(k)) for k in nodes[:n]] == [rt.cudaGraphNodeType.cudaGraphNodeTypeKernel]
    outer = ok(rt.cudaGraphCreate(0))
    ok(rt.cudaGraphAddChildGraphNode(outer, None, 0, graph))
    execs = [ok(rt.cudaGraphInstantiate(g, 0)) for g in (graph, graph, outer)]
    V, dV = nb.exact(p)
    for ex in execs:
        d_v.zero_()
        d_g.zero_()
        torch.cuda.synchronize()
        ok(rt.cudaGraphLaunch(ex, st))
        ok(rt.cudaStreamSynchronize(st))
        assert np.array_equal(d_v.cpu().numpy(), V) and np.array_equal(d_g.cpu().numpy(), dV)
    for ex in execs:
        ok(rt.cudaGraphExecDestroy(ex))
    for g in (outer, graph):
        ok(rt.cudaGraphDestroy(g))
    ok(rt.cudaStreamDestroy(st))
    nb.close()


@pytest.mark.parametrize("npts,nh", [(18944, 300), (18945, 300), (18945, 301), (20011, 1), (9472, 64), (9473, 64), (9473, 65),
                                     (1000, 12000), (1001, 12000), (700, 12001), (12000, 1000), (12001, 1000),
                                     (33, 2049)])
@pytest.mark.parametrize("D", [3, 4])
def test_sums_at_the_edges_of_the_routes(npts, nh, D):
    lo, hi = systems.CV4_LO[:D], systems.CV4_HI[:D]
    c, h, s = _hills(nh, D, npts, True)
    rng = np.random.default_rng(npts)
    p = lo + (hi - lo) * (1.2 * rng.random((npts, D)) - 0.1)
    bad = rng.choice(npts, 3, replace=False)
    p[bad, 0] = np.nan, np.inf, -np.inf
    nb = mtd.NNBias(lo, hi)
    nb.add_hills(c, h, s)
    gv, gd = nb.exact(p)
    nb.close()
    assert not np.any(gv[bad]) and not np.any(gd[bad])
    some = np.setdiff1d(np.concatenate([np.arange(40), rng.choice(npts, 400), np.arange(npts - 40, npts)]) % npts, bad)
    V, dV, aV, adV = _sum(p[some], c, h, s)
    cut = nh * np.abs(h).max() * np.exp(-40.0)
    assert np.all(np.abs(gv[some] - V) <= 1e-13 * aV + cut)
    assert np.all(np.abs(gd[some] - dV) <= 1e-13 * adV + 10 * cut / s.min())
