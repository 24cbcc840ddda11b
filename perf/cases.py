"""What this framework is timed on: one pass each of the work its users have it do.

A pass is one call of a public entry point, the way an MD program makes it:
`post_force` (host arrays) or `post_force_device` (arrays in device memory) of
a `fix metad` instance, one step of a walker group, or one batch of the learned
bias.  Sizes are those of the repository's own configurations (4,000-atom FCC
with Q6, 256,000-atom slabs with Q4 + Q6, 1,048,576 atoms x 96 k-vectors, 32
walkers, 20,000 4D hills) and of the plugin's own Q4 run (32,000 atoms), with
ordinary and odd ones between them; `draw` gives more of the same ranges.

Forces: an MD step hands over pair forces and gets them back with the bias
force taken off, so f holds N(0, 0.5 eV/A) per component, as in a metal.  The
bias grid holds the hills of a run in progress, and the first pass deposits.

`exact` restates each path in 64 bits with plain torch: neighbour pairs from a
dense cell table, the CV as a differentiable function of the positions, its
gradient by autograd, the grid in numpy.
"""
import math
import os
import sys
import tempfile

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "metad-toy_b200"))
import mtd  # noqa: E402
import systems  # noqa: E402

A = 5.26                 # FCC lattice constant (A)
KB = 8.617343e-5         # eV / K
FORCE = 0.5              # eV / A, spread of the pair forces in f
FIRST = 10               # step number of the first timed pass (PACE 10: it deposits)
PACE = 10


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest runs, where latency and launches count
        {"name": "q6_4k_fp64", "kind": "q", "nc": 10, "l": 6, "rc": 3.9, "cap": 18, "prec": "fp64", "host": False},
        {"name": "ql_4k_fp64", "kind": "ql", "n": 4000, "sw": "STEP", "skin": False, "prec": "fp64"},
        # the plugin's own benchmark deck (32,000 atoms, Q4, the cap binds), called as LAMMPS
        # calls it: host arrays in, host arrays out
        {"name": "q4_32k_host", "kind": "q", "nc": 20, "l": 4, "rc": 6.0, "cap": 12, "prec": "mixed", "host": True},
        # an ordinary system with an odd atom count and a smooth switch, lists rebuilt every step
        {"name": "ql_61k_fermi", "kind": "ql", "n": 61111, "sw": "FERMI", "skin": False, "prec": "mixed"},
        # the headline: 256,000 atoms, local Q4 + Q6, skin lists
        {"name": "ql_256k_skin", "kind": "ql", "n": 256000, "sw": "STEP", "skin": True, "prec": "mixed"},
        # k-vector structure factor: an ordinary system in FP64 and the full-size one in mixed precision
        {"name": "sk_108k_24_fp64", "kind": "sk", "nc": 30, "nk": 24, "prec": "fp64"},
        {"name": "sk_1m_96", "kind": "sk", "nc": 64, "nk": 96, "prec": "mixed"},
        # Debye structure factor, the number of ordered atoms as CV
        {"name": "debye_32k", "kind": "debye", "nc": 20, "mode": "COUNT", "prec": "mixed"},
        # many walkers of uneven size that share one grid
        {"name": "walkers_32", "kind": "walkers", "walkers": 32, "nmin": 2000, "nmax": 64000},
        # 4D bias: the exact hill sum and the network on a batch of CV points, and the network's
        # backward pass on one training batch
        {"name": "hillsum_64k", "kind": "hillsum", "npts": 65536, "hills": 20000, "dim": 4},
        {"name": "mlp_64k", "kind": "mlp", "npts": 65536, "dim": 4},
        {"name": "mlp_grad_8k", "kind": "mlp_grad", "npts": 8192, "dim": 4},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["q", "ql", "ql", "sk", "debye", "walkers", "hillsum", "mlp", "mlp_grad"])
    prec = rng.choice(["mixed", "mixed", "fp64"])
    if kind == "q":
        rc, cap = rng.choice([(3.9, 18), (6.0, 12)])
        return {"kind": kind, "nc": _log_int(rng, 7, 20), "l": rng.choice([4, 6]), "rc": rc, "cap": cap, "prec": prec,
                "host": rng.random() < 0.3}
    if kind == "ql":
        n = _log_int(rng, 3000, 256000 if prec == "mixed" else 100000)
        return {"kind": kind, "n": n, "sw": rng.choice(["STEP", "FERMI"]), "skin": rng.random() < 0.5, "prec": prec}
    if kind == "sk":
        return {"kind": kind, "nc": _log_int(rng, 16, 64 if prec == "mixed" else 34), "nk": rng.randint(12, 96),
                "prec": prec}
    if kind == "debye":
        return {"kind": kind, "nc": _log_int(rng, 7, 20), "mode": rng.choice(["AVE", "COUNT"]), "prec": prec}
    if kind == "walkers":
        nmin = _log_int(rng, 1500, 8000)
        return {"kind": kind, "walkers": rng.randint(3, 32), "nmin": nmin, "nmax": nmin + _log_int(rng, 500, 50000)}
    if kind == "hillsum":
        return {"kind": kind, "npts": _log_int(rng, 500, 65536), "hills": _log_int(rng, 1000, 20000),
                "dim": rng.choice([3, 4, 4])}
    return {"kind": kind, "npts": _log_int(rng, 300, 65536 if kind == "mlp" else 8192), "dim": rng.choice([3, 4, 4])}


# ------------------------------------------------------------------ decks and positions
def _hist(case):
    """Grid of the deck: (bins, range, hill width, height, bias factor, well-tempered)."""
    if case["kind"] == "q":
        return [1000], [(0.0, 1.0)], 0.01, 0.005, 10.0, 0
    if case["kind"] == "sk":
        return [2000], [(0.0, 10.0)], 0.05, 0.005, 10.0, 0
    if case["kind"] == "debye":
        hi = 2.0 if case["mode"] == "AVE" else 4.0 * case["nc"] ** 3
        return [400], [(0.0, hi)], hi * 0.01, 0.005, 10.0, 0
    nb = 256 if case["kind"] == "walkers" else 200
    return [nb, nb], [(0.0, 1.0), (0.0, 1.0)], 0.01, 0.005, 9.0, 1


def _deck(case):
    bins, rng, sigma, h0, biasf, wt = _hist(case)
    a = ["GAUSSIAN", sigma, h0, biasf, "PACE", PACE, "TEMP", 300.0]
    if case["kind"] == "q":
        a += ["CAL", "NAME", "Q", "STEINH", "Q", case["l"], "all", "cutoff_r", case["rc"], "cutoff_Natoms", case["cap"],
              "SYMBOL", "v1", "Q.AVE"]
    elif case["kind"] == "sk":
        a += ["CAL", "NAME", "SK", "STRU_FACTOR_K", "all", "nk", case["nk"], "kmag", systems.KMAG_111, "seed", 3,
              "SYMBOL", "v1", "SK.AVE"]
    elif case["kind"] == "debye":
        a += ["CAL", "NAME", "SF", "STRU_FACTOR", "all", "cutoff_r", 6.0, "q_factor", 2.8,
              "SW_func", "FERMI", "r_0", 1.0, "alpha", 5.0, "SYMBOL", "v1", "SF." + case["mode"]]
    else:
        fermi = case.get("sw") == "FERMI"
        a += ["CAL", "NAME", "SW", "SW_FUNC"] + (["FERMI", "r_0", 3.9, "alpha", -8.0] if fermi else ["STEP", "r_0", 3.9])
        for l in (4, 6):
            a += ["CAL", "NAME", "Q%d" % l, "STEINH", "L", l, "all", "cutoff_r", 3.9, "SW_FUNC_r", "SW"]
        a += ["SYMBOL", "v1", "Q4.MEAN_SOLID", "SYMBOL", "v2", "Q6.MEAN_SOLID"]
    a += ["CV_dim", len(bins)]
    for d, (nb, (lo, hi)) in enumerate(zip(bins, rng)):
        a += ["DIM", d + 1, lo, hi, nb, "v%d" % (d + 1)]
    a += ["WT", wt]
    if case.get("skin"):
        a += ["NEIGH_SKIN", 1.0, "NEIGH_EVERY", 10]
    return a


def _positions(case, seed):
    """Two thermal snapshots of the case's atoms (the positions of alternating steps) and the box."""
    if case["kind"] == "ql":
        n = case["n"]
        base, L = systems.walker_system(n, seed, nxy=max(5, int(round(24 * (n / 256000.0) ** (1 / 3)))))
        sigma = 0.05
    else:
        base, L = systems.fcc(case["nc"], A), np.array([case["nc"] * A] * 3)
        sigma = 0.2 if case["kind"] == "sk" else 0.15
    return [np.ascontiguousarray(systems.wrap(systems.jitter(base, sigma, seed, c), L)) for c in (0, 1)], L


def _walker_systems(case, seed):
    ns = np.random.default_rng(44).integers(case["nmin"], case["nmax"] + 1, size=case["walkers"])
    out = []
    for k, n in enumerate(ns):
        x, L = systems.walker_system(int(n), seed * 100 + k)
        out.append(([np.ascontiguousarray(systems.wrap(systems.jitter(x, 0.05, seed + k, c), L)) for c in (0, 1)], L))
    return out


def _pair_forces(n, seed):
    return np.random.default_rng(seed + 1).normal(0.0, FORCE, (n, 3))


def _history(case, cv, seed):
    """The hills of the run so far: 12 around the CV it stands at."""
    _, _, sigma, h0, _, _ = _hist(case)
    rng = np.random.default_rng(seed + 2)
    c = np.asarray(cv)[None, :] + sigma * rng.standard_normal((12, len(cv)))
    return c, h0 * rng.uniform(0.5, 1.0, 12)


def _network(seed):
    """Parameters of a network of the learned bias's size (He-style), flat."""
    rng = np.random.default_rng(seed)
    w = [rng.normal(0, math.sqrt(0.5), 512), rng.normal(0, 0.1, 128), rng.normal(0, math.sqrt(2 / 128), 128 * 128),
         rng.normal(0, 0.1, 128), rng.normal(0, math.sqrt(1 / 128), 128), [0.05]]
    return np.concatenate(w).astype(np.float32)


def _points(case, seed):
    D = case["dim"]
    lo, hi = systems.CV4_LO[:D], systems.CV4_HI[:D]
    return lo + (hi - lo) * np.random.default_rng(seed + 3).random((case["npts"], D)), lo, hi


def _hills(case, seed):
    c, h, s = systems.cv4_hills(n=case["hills"], seed=seed)
    return np.ascontiguousarray(c[:, :case["dim"]]), h, s


def _targets(p):
    return np.sin(3 * p[:, 0]) * np.cos(2 * p[:, 1]) + p[:, 2] * p[:, -1]


VSCALE = 0.7


# ------------------------------------------------------------------ prepare and run
def _again(call):
    """A call whose neighbour lists proved too small grows them and asks to be made again."""
    for _ in range(4):
        try:
            return call()
        except mtd.MetadError as e:
            if mtd.STATUS_NAMES.get(e.status) != "NEIGH_OVERFLOW":
                raise
    return call()


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("hillsum", "mlp", "mlp_grad"):
        p, lo, hi = _points(case, seed)
        nb = mtd.NNBias(lo, hi, seed=3)
        s = {"kind": kind, "nb": nb, "n": case["npts"]}
        if kind == "hillsum":
            nb.add_hills(*_hills(case, seed))
        else:
            nb.set_params(_network(seed), VSCALE)
        if kind == "mlp_grad":
            s["p"], s["t"] = p, _targets(p)
        else:
            s["p"] = torch.from_numpy(p).cuda()
            s["out"] = torch.zeros(case["npts"] * (1 + case["dim"]), dtype=torch.float64, device="cuda")
            s["stream"] = torch.cuda.Stream()
            torch.cuda.synchronize()
        return s
    if kind == "walkers":
        syss = _walker_systems(case, seed)
        W = mtd.Walkers(len(syss), _deck(case), precision="mixed")
        for k, (_, L) in enumerate(syss):
            W.set_box(k, [0, 0, 0], L)
        W.init()
        ns = [xs[0].shape[0] for xs, _ in syss]
        x = [[torch.from_numpy(xs[c]).cuda() for xs, _ in syss] for c in (0, 1)]
        f = [torch.from_numpy(_pair_forces(n, seed + k)).cuda() for k, n in enumerate(ns)]
        s = {"kind": kind, "W": W, "ns": ns, "x": x, "f": f, "step": FIRST,
             "xp": [[t.data_ptr() for t in v] for v in x], "fp": [t.data_ptr() for t in f]}
        torch.cuda.synchronize()
        scratch = [torch.zeros_like(t) for t in f]
        torch.cuda.synchronize()

        def earlier():   # the step before, on the other snapshot: the group's first hills
            W.step_device(0, ns, s["xp"][1], [t.data_ptr() for t in scratch])
            W.sync()
        _again(earlier)
        return s
    xs, L = _positions(case, seed)
    n = xs[0].shape[0]
    m = mtd.Metad(_deck(case), precision=case["prec"])
    m.set_box([0, 0, 0], L)
    m.init()
    s = {"kind": kind, "m": m, "n": n, "step": FIRST, "host": case.get("host", False)}
    dx = [torch.from_numpy(x).cuda() for x in xs]
    f0 = torch.from_numpy(_pair_forces(n, seed))
    f1 = torch.zeros((n, 3), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()

    def earlier(c):      # earlier steps of the run, without a hill
        m.post_force_device(c + 1, n, dx[c].data_ptr(), f1.data_ptr(), f1.data_ptr())
        m.sync()
    for c in (1, 0):
        _again(lambda: earlier(c))
    centres, heights = _history(case, m.cv, seed)
    sigma = _hist(case)[2]
    with tempfile.TemporaryDirectory() as d:
        path = os.path.join(d, "HILLS")
        with open(path, "w") as fh:
            for t, (c, h) in enumerate(zip(centres, heights)):
                fh.write("%d %s %.17g %.17g\n" % (t, " ".join("%.17g" % v for v in c), h, sigma))
        m.hills_replay(path)
    if s["host"]:
        s["keep"] = [torch.from_numpy(x).pin_memory() for x in xs] + [f0.pin_memory()]
        s["x"] = [t.numpy() for t in s["keep"][:2]]
        s["f"] = s["keep"][2].numpy()
    else:
        s["x"], s["f"], s["out"] = dx, f0.cuda(), f1
    torch.cuda.synchronize()
    return s


def run(s):
    kind = s["kind"]
    if kind == "mlp_grad":       # one training batch, host arrays as the trainer samples them
        g, loss = s["nb"].loss_grad(s["p"], s["t"], VSCALE)
        return g, np.float32(loss)
    if kind in ("hillsum", "mlp"):
        v = s["out"].data_ptr()
        st = s["stream"]
        s["nb"].eval_device(s["n"], s["p"].data_ptr(), v, v + 8 * s["n"], use_nn=int(kind == "mlp"),
                            stream=st.cuda_stream)
        if kind == "hillsum":
            return s["out"]
        with torch.cuda.stream(st):
            return s["out"].float()   # the network works in FP32: its values are taken as such
    c = s["step"] & 1
    if kind == "walkers":        # the group's step ends with its outputs collected
        s["W"].step_device(s["step"], s["ns"], s["xp"][c], s["fp"])
        s["W"].sync()
        s["step"] += 1
        return s["f"]
    if s["host"]:                # f -= dV/dx in place, CVs for the thermo output
        s["m"].post_force(s["step"], s["x"][c], s["f"])
        s["step"] += 1
        return s["f"], s["m"].cv.astype(np.float32)
    s["m"].post_force_device(s["step"], s["n"], s["x"][c].data_ptr(), s["f"].data_ptr(), s["out"].data_ptr())
    s["step"] += 1
    return s["out"]


# ------------------------------------------------------------------ work
def work(case):
    kind = case["kind"]
    if kind in ("hillsum", "mlp", "mlp_grad"):
        n, D = case["npts"], case["dim"]
        if kind == "hillsum":    # distance, exponential and gradient of the hills in reach of a point
            return {"bytes": 8 * n * (2 * D + 1) + 8 * (D + 2) * case["hills"], "flops": n * case["hills"] * (3 * D + 1)}
        layer = 2 * 128 * 128 + 4 * 128 * D
        if kind == "mlp":
            return {"bytes": 8 * n * (2 * D + 1) + 4 * 17281, "flops": 2 * n * layer}
        return {"bytes": 8 * n * (D + 1) + 8 * 17281, "flops": 3 * n * layer}
    if kind == "sk":
        n = 4 * case["nc"] ** 3
        return {"bytes": 72 * n, "flops": 2.0 * n * case["nk"] * 33}
    if kind == "walkers":
        n = case["walkers"] * 0.5 * (case["nmin"] + case["nmax"])
        return {"bytes": 72 * n, "flops": n * 8 * 900}
    if kind == "ql":
        nbar = 8 if case["sw"] == "STEP" else 20
        return {"bytes": 72 * case["n"], "flops": case["n"] * nbar * 900}
    n = 4 * case["nc"] ** 3
    if kind == "debye":
        return {"bytes": 72 * n, "flops": n * 25 * 90}
    return {"bytes": 72 * n, "flops": n * 12 * 400}


# ------------------------------------------------------------------ 64-bit restatement
DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _pairs(x, L, rc):
    """All ordered pairs (i, j) with |x_j - x_i| <= rc in the periodic box, and x_j - x_i - image."""
    n = x.shape[0]
    nc = torch.clamp((L / (rc + 1e-6)).floor().long(), min=1)
    if int(nc.min()) < 3:
        raise ValueError("box below three cutoffs")
    cell = torch.minimum((x / L * nc).floor().long().clamp(min=0), nc - 1)
    flat = (cell[:, 0] * nc[1] + cell[:, 1]) * nc[2] + cell[:, 2]
    order = torch.argsort(flat, stable=True)
    ncell = int(nc.prod())
    count = torch.bincount(flat, minlength=ncell)
    start = torch.cumsum(count, 0) - count
    most = int(count.max())
    table = torch.full((ncell, most), -1, dtype=torch.long, device=x.device)
    table[flat[order], torch.arange(n, device=x.device) - start[flat[order]]] = order
    off = torch.stack(torch.meshgrid(*[torch.arange(-1, 2, device=x.device)] * 3, indexing="ij"), -1).reshape(-1, 3)
    ii, jj = [], []
    step = max(1, 20_000_000 // (27 * most))
    for a in range(0, n, step):
        i = torch.arange(a, min(n, a + step), device=x.device)
        c = (cell[i][:, None, :] + off) % nc
        j = table[(c[..., 0] * nc[1] + c[..., 1]) * nc[2] + c[..., 2]].reshape(len(i), -1)
        d = x[j.clamp(min=0)] - x[i][:, None]
        d = d - L * torch.round(d / L)
        ok = (j >= 0) & (j != i[:, None]) & ((d * d).sum(-1) <= rc * rc)
        k = ok.nonzero()
        ii.append(i[k[:, 0]])
        jj.append(j[k[:, 0], k[:, 1]])
    i, j = torch.cat(ii), torch.cat(jj)
    d = x[j] - x[i]
    return i, j, L * torch.round(d / L)


def _ylm(l, d):
    """Re and Im of Y_lm, m = 0..l, from the derivatives of the Legendre polynomial."""
    r = d.square().sum(-1).sqrt()
    u = d / r[:, None]
    wr, wi = torch.ones_like(r), torch.zeros_like(r)
    poly = np.polynomial.legendre.leg2poly([0] * l + [1])
    out = []
    for m in range(l + 1):
        norm = (-1) ** m * math.sqrt((2 * l + 1) / (4 * math.pi) * math.factorial(l - m) / math.factorial(l + m))
        v = torch.full_like(r, poly[-1])
        for c in poly[-2::-1]:
            v = v * u[:, 2] + c
        out += [norm * v * wr, norm * v * wi]
        wr, wi = wr * u[:, 0] - wi * u[:, 1], wr * u[:, 1] + wi * u[:, 0]
        poly = np.polynomial.polynomial.polyder(poly)
    return torch.stack(out, -1), r


def _norm_q(q, l):
    w = torch.full((2 * (l + 1),), 2.0, dtype=q.dtype, device=q.device)
    w[:2] = 1.0
    s = 4 * math.pi / (2 * l + 1) * (q * q * w).sum(-1)
    ok = s > 0
    return torch.where(ok, torch.where(ok, s, torch.ones_like(s)).sqrt(), torch.zeros_like(s))


def _cvs(case, x, L):
    """The deck's CVs as differentiable functions of x."""
    n = x.shape[0]
    if case["kind"] == "sk":
        k = torch.from_numpy(systems.kvectors(case["nk"], systems.KMAG_111, 3)).to(x.device)
        re, im = [], []
        for a in range(0, case["nk"], 8):
            ph = x @ k[a:a + 8].T
            re.append(ph.cos().sum(0))
            im.append(ph.sin().sum(0))
        re, im = torch.cat(re), torch.cat(im)
        return [(re * re + im * im).mean() / n]
    x0 = x.detach()
    if case["kind"] == "q":
        i, j, img = _pairs(x0, L, case["rc"])
        r2 = (x0[j] - x0[i] - img).square().sum(-1)
        o = torch.argsort(r2, stable=True)
        o = o[torch.argsort(i[o], stable=True)]
        i, j, img = i[o], j[o], img[o]
        count = torch.bincount(i, minlength=n)
        keep = torch.arange(len(i), device=x.device) - (torch.cumsum(count, 0) - count)[i] < case["cap"]
        i, j, img = i[keep], j[keep], img[keep]
        nk = torch.bincount(i, minlength=n).clamp(min=1).double()
        y, _ = _ylm(case["l"], x[j] - x[i] - img)
        q = torch.zeros((n, y.shape[1]), dtype=x.dtype, device=x.device).index_add(0, i, y) / nk[:, None]
        return [_norm_q(q, case["l"]).mean()]
    if case["kind"] == "debye":
        i, j, img = _pairs(x0, L, 6.0)
        r = (x[j] - x[i] - img).square().sum(-1).sqrt()
        t = ((r * r - 0.8 * 36.0) / (0.2 * 36.0)).clamp(min=0)
        S = 1.0 + torch.zeros(n, dtype=x.dtype, device=x.device).index_add(
            0, i, torch.sin(2.8 * r) / (2.8 * r) * (1 - t * t * t))
        return [S.mean() if case["mode"] == "AVE" else (1 / (1 + torch.exp(-5.0 * (S - 1.0)))).sum()]
    fermi = case.get("sw") == "FERMI"
    # neighbours of a smooth switch: where it is at least cutoff_eps (1e-6)
    i, j, img = _pairs(x0, L, 3.9 + math.log(1e6 - 1) / 8.0 if fermi else 3.9)
    d = x[j] - x[i] - img
    r0 = d.detach().square().sum(-1).sqrt()
    if not fermi:
        on = r0 < 3.9
        i, j, d = i[on], j[on], d[on]
    out = []
    for l in (4, 6):
        y, r = _ylm(l, d)
        sg = 1 / (1 + torch.exp(8.0 * (r - 3.9))) if fermi else torch.ones_like(r)
        nf = torch.zeros(n, dtype=x.dtype, device=x.device).index_add(0, i, sg)
        z = torch.zeros((n, y.shape[1]), dtype=x.dtype, device=x.device)
        q = z.index_add(0, i, sg[:, None] * y) / torch.where(nf > 0, nf, torch.ones_like(nf))[:, None]
        lq = (q + z.index_add(0, i, sg[:, None] * q[j])) / (nf + 1)[:, None]
        out.append(_norm_q(lq, l).mean())
    return out


class _Grid:
    """The bias grid: hills deposited within their band, Catmull-Rom interpolation."""

    def __init__(self, case):
        self.bins, self.range, self.sigma, self.h0, self.biasf, self.wt = _hist(case)
        self.g = np.zeros(self.bins)
        self.d = [(hi - lo) / nb for nb, (lo, hi) in zip(self.bins, self.range)]

    def add(self, s, w):
        sl, r2 = [], 0.0
        for k, (nb, (lo, _), d) in enumerate(zip(self.bins, self.range, self.d)):
            R, c = int(math.ceil(4 * self.sigma / d)) + 1, int((s[k] - lo) / d)
            a, b = max(0, c - R), min(nb - 1, c + R)
            sl.append(slice(a, b + 1))
            e = (s[k] - (lo + (np.arange(a, b + 1) + 0.5) * d)) ** 2
            r2 = e if k == 0 else r2[:, None] + e[None, :]
        self.g[tuple(sl)] += w * np.exp(-0.5 * r2 / self.sigma ** 2)

    def value(self, s):
        def weights(f):
            v = np.array([-0.5 * f + f * f - 0.5 * f ** 3, 1 - 2.5 * f * f + 1.5 * f ** 3,
                          0.5 * f + 2 * f * f - 1.5 * f ** 3, -0.5 * f * f + 0.5 * f ** 3])
            return v, np.array([-0.5 + 2 * f - 1.5 * f * f, -5 * f + 4.5 * f * f, 0.5 + 4 * f - 4.5 * f * f,
                                -f + 1.5 * f * f])
        sl, w, dw = [], [], []
        for k, (nb, (lo, _), d) in enumerate(zip(self.bins, self.range, self.d)):
            u = (s[k] - lo) / d - 0.5
            i = int(math.floor(u))
            f = u - i
            if i < 1:
                i, f = 1, 0.0
            if i > nb - 3:
                i, f = nb - 3, 1.0
            a, b = weights(f)
            sl.append(slice(i - 1, i + 3))
            w.append(a)
            dw.append(b / d)
        p = self.g[tuple(sl)]
        if len(w) == 1:
            return float(p @ w[0]), [float(p @ dw[0])]
        return float(w[0] @ p @ w[1]), [float(dw[0] @ p @ w[1]), float(w[0] @ p @ dw[1])]

    def height(self, s):
        return self.h0 * math.exp(-(self.value(s)[0] if self.wt else 0.0) / (300.0 * KB * (self.biasf - 1.0)))


def _values(case, x, L):
    with torch.no_grad():
        return [float(c) for c in _cvs(case, torch.from_numpy(x).to(DEV), torch.from_numpy(L).to(DEV))]


def _forces(case, x, L, dV, f):
    x = torch.from_numpy(x).to(DEV).requires_grad_(True)
    g, = torch.autograd.grad(sum(v * c for v, c in zip(dV, _cvs(case, x, torch.from_numpy(L).to(DEV)))), x)
    return torch.from_numpy(f).to(DEV) - g


def _sk_forces(case, x, dV, f):
    """S(k) without autograd's stored phases: the closed form, 8 k-vectors at a time."""
    x = torch.from_numpy(x).to(DEV)
    k = torch.from_numpy(systems.kvectors(case["nk"], systems.KMAG_111, 3)).to(DEV)
    g = torch.zeros_like(x)
    for a in range(0, case["nk"], 8):
        ph = x @ k[a:a + 8].T
        s, c = ph.sin(), ph.cos()
        g += (c * s.sum(0) - s * c.sum(0)) @ k[a:a + 8]
    return torch.from_numpy(f).to(DEV) - dV * 2.0 / (x.shape[0] * case["nk"]) * g


def _silu(z):
    s = torch.sigmoid(z)
    return z * s


def _net(w, u):
    W1, b1, W2 = w[:512].reshape(128, 4), w[512:640], w[640:17024].reshape(128, 128)
    b2, w3, b3 = w[17024:17152], w[17152:17280], w[17280]
    return _silu(_silu(u @ W1.T + b1) @ W2.T + b2) @ w3 + b3


def _exact_net(case, seed):
    """The network in 64 bits on its BF16 weights, activations unrounded."""
    p, lo, hi = _points(case, seed)
    w32 = torch.from_numpy(_network(seed))
    w = w32.double()
    for a, b in ((0, 512), (640, 17024), (17152, 17280)):
        w[a:b] = w32[a:b].bfloat16().double()
    w = w.to(DEV)
    u = torch.zeros((case["npts"], 4), dtype=torch.float64, device=DEV)
    u[:, :case["dim"]] = torch.from_numpy(2.0 * (p - lo) / (hi - lo) - 1.0).to(DEV)
    if case["kind"] == "mlp":
        u.requires_grad_(True)
        y = _net(w, u)
        g, = torch.autograd.grad(y.sum(), u)
        sc = torch.from_numpy(2.0 / (hi - lo)).to(DEV)
        return torch.cat([VSCALE * y.detach(), (VSCALE * g[:, :case["dim"]] * sc).reshape(-1)])
    w.requires_grad_(True)
    t = torch.from_numpy(_targets(p) / VSCALE).to(DEV)
    loss = (_net(w, u) - t).square().mean()
    g, = torch.autograd.grad(loss, w)
    return g.cpu().numpy(), np.float64(loss.detach().cpu())


def exact(case, seed):
    kind = case["kind"]
    if kind in ("mlp", "mlp_grad"):
        return _exact_net(case, seed)
    if kind == "hillsum":
        p = torch.from_numpy(_points(case, seed)[0]).to(DEV)
        c, h, s = (torch.from_numpy(v).to(DEV) for v in _hills(case, seed))
        V, G = [], []
        for a in range(0, len(p), 512):
            d = p[a:a + 512, None, :] - c
            e = h * torch.exp(-0.5 * d.square().sum(-1) / (s * s))
            V.append(e.sum(1))
            G.append(-(e[..., None] * d / (s * s)[:, None]).sum(1))
        return torch.cat([torch.cat(V), torch.cat(G).reshape(-1)])
    grid = _Grid(case)
    if kind == "walkers":
        syss = _walker_systems(case, seed)
        for c in (1, FIRST & 1):     # the step before, then the timed one
            cvs = [_values(case, xs[c], L) for xs, L in syss]
            for s, w in [(s, grid.height(s)) for s in cvs]:
                grid.add(s, w)
        out = []
        for k, ((xs, L), s) in enumerate(zip(syss, cvs)):
            x = xs[FIRST & 1]
            out.append(_forces(case, x, L, grid.value(s)[1], _pair_forces(x.shape[0], seed + k)))
        return out
    xs, L = _positions(case, seed)
    x = xs[FIRST & 1]
    cv = _values(case, x, L)
    for c, h in zip(*_history(case, _values(case, xs[0], L), seed)):
        grid.add(c, h)
    grid.add(cv, grid.height(cv))
    dV = grid.value(cv)[1]
    f = _pair_forces(x.shape[0], seed)
    if kind == "sk":
        return _sk_forces(case, x, dV[0], f)
    f = _forces(case, x, L, dV, f)
    return (f.cpu().numpy(), np.array(cv)) if case.get("host") else f
