"""The calls whose time this framework answers for, through its public Python entry points.

Six kinds of work, each over the range of sizes that its users have:

* ``pack``: one packing advanced by ``run_packing_observed`` from host arrays (set-up, ``max_steps`` steps of the
  relaxation loop, results back on the host): what ``Packing.pack`` and ``Packing.relax`` do. Particles are placed by
  ``initialize_particles``, as a user's are. Runs are capped, because a relaxation amplifies rounding: over
  many thousands of steps two correct engines end in different jammed states.
* ``batch``: many packings in one ``run_packing_batch`` call, drawn like the batched workload of ``bench.py``.
* ``overlap``: ``jobs.overlap_report`` of a state on the host (the analysis of a study's packings).
* ``train`` and ``predict``: the warm start's network, one optimizer step in mid-training and the prediction for
  a list of packings.

``draw`` gives further cases of the same ranges.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import rcpgenerator_b200 as rb
from rcpgenerator_b200 import jobs
from rcpgenerator_b200 import warmstart as W

# ---- the cases -------------------------------------------------------------------------


def _pack(name, n, nd, dist, steps, **kw):
    c = {"name": name, "kind": "pack", "n": n, "ndim": nd, "dist": dist, "steps": steps, "precision": "f64",
         "engine": "graph", "walls": "none", "side": 1.0}
    c.update(kw)
    return c


def listed():
    return [
        # the smallest packing of the batched workload, run by itself: launches and the serial controller
        _pack("pack_2d_n64", 64, 2, "mono", 3000),
        # the reference's own example, 3-D monodisperse spheres, N = 2,000
        _pack("pack_3d_n2000", 2000, 3, "mono", 1500),
        # the same in the bit-for-bit engine, as a user checks results against the reference
        _pack("pack_exact_3d_n2000", 2000, 3, "mono", 96, engine="exact"),
        # a large packing of the batched workload in four dimensions, mixed precision
        _pack("pack_4d_n12001", 12001, 4, "lognormal", 250, precision="mixed"),
        # 2-D disks between hard walls, an ordinary size with an odd count. Steps are absolute lengths: in a box of
        # side 20 they are short against the disks and few of them rebuild the neighbour rows, as over most of a run
        _pack("pack_walls_2d_n25003", 25003, 2, "bidisperse", 1200, walls="flat", side=20.0),
        # the size at which the warm start is evaluated, FP64 pair arithmetic
        _pack("pack_3d_n100000", 100_000, 3, "bidisperse", 400),
        # a wide power law in a spherical container (size classes), mixed precision
        _pack("pack_powerlaw_3d_n300007", 300_007, 3, "powerlaw", 64, precision="mixed", walls="sphere"),
        # the benchmark's packing: a million bidisperse disks, mixed precision
        _pack("pack_2d_n1000000", 1_000_000, 2, "bidisperse", 600, precision="mixed"),
        # a study: packings of uneven size and dimension in one call
        {"name": "batch_96", "kind": "batch", "count": 96, "n_max": 4096, "steps": 400, "precision": "mixed"},
        # overlap diagnostics of one large packed state
        {"name": "overlap_3d_n200003", "kind": "overlap", "n": 200_003, "ndim": 3, "dist": "bidisperse"},
        # one optimizer step of the warm start's training at its default batch
        {"name": "train_b256", "kind": "train", "batch": 256},
        # growth lengths for every packing of the batched workload
        {"name": "predict_b4096", "kind": "predict", "batch": 4096},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pack", "pack", "pack", "pack", "batch", "overlap", "train", "predict"])
    if kind == "pack":
        engine = rng.choice(["graph"] * 7 + ["exact"])
        nd = rng.choice([2, 2, 3, 3, 4])
        n = _log(rng, 64, 3000 if engine == "exact" else {2: 700_000, 3: 120_000, 4: 12_000}[nd])
        dist = rng.choice(["mono", "bidisperse", "lognormal"] + (["powerlaw"] if nd == 3 and n < 60_000 else []))
        walls = rng.choice(["none", "none", "none", "flat"] + (["sphere"] if nd == 3 else []))
        # larger packings get fewer steps, so that no drawn case costs more than the largest listed one
        work = n * {2: 1.0, 3: 6.0, 4: 40.0}[nd] * (4.0 if dist in ("lognormal", "powerlaw") else 1.0)
        steps = 48 if engine == "exact" else max(32, min(1000, int(2.0e8 / work)))
        return {"kind": "pack", "n": n, "ndim": nd, "dist": dist, "steps": steps, "walls": walls, "engine": engine,
                "side": rng.choice([1.0, 1.0, 5.0, 20.0]), "precision": "f64" if engine == "exact" else rng.choice(["f64", "mixed"])}
    if kind == "batch":
        return {"kind": "batch", "count": _log(rng, 8, 90), "n_max": _log(rng, 500, 4000),
                "steps": rng.randrange(200, 400), "precision": rng.choice(["f64", "mixed"])}
    if kind == "overlap":
        return {"kind": "overlap", "n": _log(rng, 500, 180_000), "ndim": rng.choice([2, 3]),
                "dist": rng.choice(["mono", "bidisperse", "uniform"])}
    return {"kind": kind, "batch": _log(rng, 1 if kind == "predict" else 16, 4096 if kind == "predict" else 1024)}


# ---- inputs ------------------------------------------------------------------------------


def _dist(kind, n, rng):
    if kind == "mono":
        return {"type": "mono", "d": 1.0}
    if kind == "bidisperse":
        return {"type": "bidisperse", "d1": 1.0, "d2": 1.4, "p": 0.5}
    if kind == "powerlaw":
        return {"type": "powerlaw", "d_min": 0.1, "d_max": 1.0, "exponent": -3.0}
    s2 = math.log1p(0.3 * 0.3)  # log-normal of std/mean 0.3, truncated like the batched workload's
    d = rng.lognormal(-0.5 * s2, math.sqrt(s2), size=2 * n + 64)
    return {"type": "custom", "custom": d[(d >= 0.2) & (d <= 5.0)][:n]}


_PHI = {2: 0.30, 3: 0.15, 4: 0.08}


def _state(case, seed):
    """Positions, diameters, box and walls as the initializer places them."""
    nd, n = case["ndim"], case["n"]
    walls = {"none": [0] * nd, "flat": [1] * nd, "sphere": [-nd] + [0] * (nd - 1)}[case.get("walls", "none")]
    init = rb.initialize_particles({"phi": _PHI[nd], "N": n, "Ndim": nd, "box": [case["side"]] * nd, "walls": walls,
                                    "dist": _dist(case["dist"], n, np.random.default_rng(seed)), "seed": seed})
    inp = {"positions": np.asarray(init["positions"]), "diameters": np.asarray(init["diameters"])}
    return inp, {"box": init["box"], "walls": init["walls"], "neighbor_max": 0, "seed": seed}


class _Packed:
    """What overlap_report looks at: a packing's positions, diameters and box."""

    def __init__(self, positions, diameters, box):
        self.positions, self.diameters, self.box = positions, diameters, box


def _overlap_state(case, seed):
    """A disordered contact network: a jittered grid whose nearest sites all overlap (2 d contacts per particle, as in
    a packing at jamming) and whose diagonal ones do not, particles in random order."""
    rng = np.random.default_rng(seed)
    n, nd = case["n"], case["ndim"]
    side = math.ceil(n ** (1.0 / nd))
    site = rng.permutation(n)
    grid = np.stack([(site // side ** k) % side for k in range(nd)], axis=1)
    pos = (grid + 0.5 + rng.uniform(-0.02, 0.02, (n, nd))) / side
    d = {"mono": np.full(n, 1.15), "bidisperse": rng.permutation(np.where(np.arange(n) % 2 == 0, 1.06, 1.22))}
    d = d.get(case["dist"], rng.uniform(1.06, 1.22, n))
    d[0] = 1.22 if case["dist"] != "mono" else d[0]
    return pos, d / side, [1.0] * nd


def _batch_items(case, seed):
    """Packings of the batched workload's kinds. Sizes, dimensions and distributions belong to the case, the particles'
    places and diameters to the seed."""
    rng = np.random.default_rng(case["count"] * 100_003 + case["n_max"])
    items = []
    for k in range(case["count"]):
        n = int(round(math.exp(rng.uniform(math.log(64), math.log(case["n_max"])))))
        c = {"n": n, "ndim": int(rng.integers(2, 5)), "side": 1.0,
             "dist": str(rng.choice(["mono", "bidisperse", "lognormal"]))}
        inp, cfg = _state(c, seed * 4096 + k)
        items.append((inp, dict(cfg, pair_precision=case["precision"])))
    return items


def _net_arrays(case, seed):
    """The warm start's network in mid-training: weights, Adam moments, a batch of standardised rows."""
    rng = np.random.default_rng(seed)
    parts = []
    for i, o in zip(W.WIDTHS[:-1], W.WIDTHS[1:]):
        parts += [rng.normal(0.0, math.sqrt(2.0 / i), o * i), rng.normal(0.0, 0.05, o)]
    w = np.concatenate(parts).astype(np.float32)
    m = (1e-3 * rng.standard_normal(w.size)).astype(np.float32)
    v = (1e-5 * rng.uniform(0.5, 2.0, w.size)).astype(np.float32)
    x = rng.standard_normal((case["batch"], W.WIDTHS[0])).astype(np.float32)
    t = rng.standard_normal((case["batch"], W.WIDTHS[-1])).astype(np.float32)
    ow = np.ones(W.WIDTHS[-1], np.float32)
    ow[0] = 4.0
    return w, m, v, x, t, ow


_TRAIN_STEP, _LR = 1000, 1e-3


def _raw_descriptors(case, seed):
    """Descriptor rows like those of the batched workload's packings."""
    rng = np.random.default_rng(seed)
    b = case["batch"]
    nd = rng.integers(2, 5, b)
    cv = rng.uniform(0.0, 0.6, b)
    k = np.arange(1, 9)
    mom = 0.5 * np.log1p(cv[:, None] ** 2) * (k - 1)[None, :]  # log-normal moments: log(m_k) / k
    log_n = rng.uniform(math.log(64), math.log(16384), b)
    return np.concatenate([mom, nd[:, None], np.zeros((b, 2)), log_n[:, None]], axis=1)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "pack":
        inp, cfg = _state(case, seed)
        cfg.update(engine=case["engine"], pair_precision=case["precision"])
        return {"kind": kind, "input": inp, "config": cfg, "options": {"max_steps": case["steps"]}}
    if kind == "batch":
        items = _batch_items(case, seed)
        return {"kind": kind, "items": items, "options": {"max_steps": case["steps"]}}
    if kind == "overlap":
        return {"kind": kind, "packing": _Packed(*_overlap_state(case, seed))}
    if kind == "train":
        w, m, v, x, t, ow = _net_arrays(case, seed)
        net = W.Network(params=w)
        net.m.copy_(torch.from_numpy(m))
        net.v.copy_(torch.from_numpy(v))
        net.step = _TRAIN_STEP - 1
        return {"kind": kind, "net": net, "x": net._dev(x), "t": net._dev(t), "ow": net._dev(ow)}
    return {"kind": kind, "ws": W.WarmStart.load(), "x": _raw_descriptors(case, seed)}


# ---- one pass ----------------------------------------------------------------------------

_FIELDS = ("positions", "diameters", "phi_history", "force_history", "energy_history", "max_overlap_history",
           "mu_history", "alpha_history")


def run(state):
    kind = state["kind"]
    if kind == "pack":
        r = rb.run_packing_observed(state["input"], state["config"], options=state["options"], as_arrays=True)["result"]
        out = {k: r[k] for k in _FIELDS}
        out.update(particle_origin=r["particle_origin"].view(np.int64), steps=r["steps"], phi=r["phi"])
        return out
    if kind == "batch":
        rs = rb.run_packing_batch(state["items"], state["options"])
        out = {k: np.concatenate([r[k].ravel() for r in rs]) for k in _FIELDS}
        out["particle_origin"] = np.concatenate([r["particle_origin"].view(np.int64) for r in rs])
        out["steps"] = np.array([r["steps"] for r in rs])
        return out
    if kind == "overlap":
        return jobs.overlap_report(state["packing"])
    if kind == "train":
        net = state["net"]
        loss = net.train_step(state["x"], state["t"], _LR, state["ow"])
        return {"loss": loss, "grad": net.grad, "weights": net.w32, "m": net.m, "v": net.v}
    return state["ws"].predict(state["x"])


# ---- what a pass cannot do without ---------------------------------------------------------


def work(case):
    kind = case["kind"]
    if kind in ("pack", "batch"):
        if kind == "pack":
            n, nd, steps = case["n"], float(case["ndim"]), case["steps"]
        else:  # N log-uniform on [64, n_max], three dimensions on average
            n, nd, steps = case["count"] * (case["n_max"] - 64) / math.log(case["n_max"] / 64), 3.0, case["steps"]
        # per step and particle: position, diameter, moments and force read, position, moments and force
        # written (FP64), and a row of about 2^(d+1) contacts and near neighbours
        row = 2.0 ** (nd + 1)
        return {"bytes": n * steps * (8.0 * (6 * nd + 1) + 4.0 * row), "flops": n * steps * (row * (5 * nd + 5) + 20 * nd)}
    if kind == "overlap":
        n, nd = case["n"], case["ndim"]
        return {"bytes": n * (8.0 * (nd + 1) + 3.0 * nd * 24.0), "flops": n * 4.0 ** nd * (4.0 * nd)}
    mults = sum(i * o for i, o in zip(W.WIDTHS[:-1], W.WIDTHS[1:]))
    if kind == "train":
        return {"bytes": mults * (2.0 + 4.0 * 7.0) + case["batch"] * 4.0 * (W.WIDTHS[0] + W.WIDTHS[-1]),
                "flops": 6.0 * mults * case["batch"]}
    return {"bytes": mults * 2.0 + case["batch"] * 8.0 * (W.WIDTHS[0] + W.WIDTHS[-1]), "flops": 2.0 * mults * case["batch"]}


# ---- the same in 64 bits ---------------------------------------------------------------------


def _layers(w):
    o, out = 0, []
    for i, n in zip(W.WIDTHS[:-1], W.WIDTHS[1:]):
        out.append((w[o:o + n * i].reshape(n, i), w[o + n * i:o + n * i + n]))
        o += n * i + n
    return out


def _net64(w, x):
    for k, (a, b) in enumerate(_layers(w)):
        x = x @ a.T + b
        if k < len(W.WIDTHS) - 2:
            x = torch.nn.functional.gelu(x)
    return x


def _exact_overlap(case, seed):
    pos, d, box = _overlap_state(case, seed)
    x = torch.from_numpy(pos).cuda()
    r = torch.from_numpy(np.asarray(d)).cuda() / 2.0
    L = torch.tensor(box, dtype=torch.float64, device="cuda")
    rq, cand, hits = 2.0 * float(r.max()), 0, []
    for i0 in range(0, len(x), 512):
        s = torch.zeros((min(512, len(x) - i0), len(x) - i0), dtype=torch.float64, device="cuda")
        for k in range(x.shape[1]):
            dd = x[i0:i0 + 512, None, k] - x[None, i0:, k]
            dd -= torch.round(dd / L[k]) * L[k]
            s += dd * dd
        near = torch.nonzero(s.sqrt_() <= rq)
        near = near[near[:, 1] > near[:, 0]]
        cand += len(near)
        dist = s[near[:, 0], near[:, 1]]
        ri, rj = r[i0 + near[:, 0]], r[i0 + near[:, 1]]
        ov = ri + rj - dist
        m = ov > 0
        hits.append((i0 + near[m], ov[m] / (ri + rj)[m], ov[m] / torch.minimum(ri, rj)[m]))
    pairs, fs, fm = (torch.cat(v) for v in zip(*hits))
    big = float(fs.max()) if len(fs) else 0.0
    return {"n_overlapping": len(fs), "n_candidate_pairs": cand, "fractions_min": fm, "fractions_sum": fs,
            "max_overlap": big, "mean_overlap": float(fs.mean()) if len(fs) else 0.0, "X_shrink_to_clear": big,
            "ndim": case["ndim"], "pairs": pairs}


def exact(case, seed):
    kind = case["kind"]
    if kind == "overlap":
        return _exact_overlap(case, seed)
    if kind == "train":
        w, m, v, x, t, ow = (torch.from_numpy(a).cuda().double() for a in _net_arrays(case, seed))
        w.requires_grad_(True)
        terms = ow * (_net64(w, x) - t) ** 2
        loss = terms.sum() / terms.numel()
        (g,) = torch.autograd.grad(loss, w)
        m = 0.9 * m + 0.1 * g
        v = 0.999 * v + 0.001 * g * g
        step = _LR * (m / (1.0 - 0.9 ** _TRAIN_STEP)) / ((v / (1.0 - 0.999 ** _TRAIN_STEP)).sqrt() + 1e-8)
        return {"loss": loss.detach(), "grad": g, "weights": (w - step).detach(), "m": m, "v": v}
    if kind == "predict":
        z = np.load(W.MODEL_PATH, allow_pickle=False)
        x = np.clip(_raw_descriptors(case, seed), z["x_lo"], z["x_hi"])
        x = torch.from_numpy((x - z["x_mean"]) / z["x_std"]).cuda()
        y = _net64(torch.from_numpy(z["params"].astype(np.float64)).cuda(), x).cpu().numpy()
        return y * z["y_std"] + z["y_mean"]
    return None  # a relaxation in 64 bits is the engine itself
