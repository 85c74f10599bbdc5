"""The calls this framework is timed on, over the sizes its users have.

listed() are the fixed cases, draw(rng) more of the same ranges; prepare()
makes what a program holds before the call, run() is one call through the
public entry points, exact() the same result in plain 64-bit torch where that
takes seconds.  Series are the package's own generators: random walks, with or
without planted motif pairs, and ECG-like pulse trains.
"""
from __future__ import annotations

import ctypes
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(
    ROOT, "scaling-subsequence-similarity-join-based-on-dynamic-time-warping-cpu-gpu_b200")


def _module(name, path, pkg_dir=None):
    if name not in sys.modules:
        spec = importlib.util.spec_from_file_location(
            name, path, submodule_search_locations=[pkg_dir] if pkg_dir else None)
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


def _dtwj():
    return _module("dtwj", os.path.join(PKG, "__init__.py"), PKG)


def _synth():
    return _module("dtwj_synth", os.path.join(PKG, "synth.py"))


def listed():
    return [
        # the smallest join of a stream of short records: latency and launches
        dict(name="join_ecg_2k", op="join", kind="ecg", n=2000, m=64, w=4, motifs=0, where="host"),
        # the CPU-runnable configuration: 20,000 samples, narrow band
        dict(name="join_walk_20k", op="join", kind="walk", n=20000, m=256, w=3, motifs=0,
             where="host"),
        # a one-shot call (the reference's seam: no context kept), ragged size,
        # quasi-periodic data on which many pairs reach DTW
        dict(name="join_ecg_9k_oneshot", op="join", kind="ecg", n=9001, m=200, w=20, motifs=0,
             where="oneshot"),
        # wide bands: ECG-like at w = 52, where DTW dominates
        dict(name="join_ecg_16k", op="join", kind="ecg", n=16384, m=512, w=52, motifs=0,
             where="host"),
        # the band sweep's random walk at ratio 0.2, ragged, already on the device
        dict(name="join_walk_131k_wide", op="join", kind="walk", n=131071, m=512, w=103, motifs=0,
             where="device"),
        # learned tile order at the shape the committed network was trained for
        dict(name="join_learned_262k", op="join", kind="walk", n=262144, m=256, w=13, motifs=8,
             where="learned"),
        # the benchmark's join: 1M samples, one planted motif pair
        dict(name="join_motif_1m", op="join", kind="walk", n=1000000, m=1024, w=52, motifs=1,
             where="device"),
        # many records of uneven length and three window lengths in one call
        dict(name="batch_48", op="batch", count=48, lo=2000, hi=32768),
        # the ED matrix profile as an output of its own
        dict(name="profile_100k", op="profile", n=100003, m=256),
        # verification of candidate pairs, FP64, from host arrays
        dict(name="pairs_host_20k", op="pairs", n=30011, m=512, w=52, count=20000, precise=1,
             where="host"),
        # a latency-bound loop that re-ranks a few pairs on the device, FP32
        dict(name="pairs_device_2k", op="pairs", n=20000, m=128, w=7, count=2000, precise=0,
             where="device"),
        # a training run of the tile network: forward, backward and Adam steps
        dict(name="mlp_train", op="train", rows=8192, epochs=8),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choices(["join", "batch", "profile", "pairs", "train"], [12, 2, 2, 3, 1])[0]
    if op == "join":
        if rng.random() < 0.4:  # ECG-like: DTW-heavy, so shorter series at long windows
            m = rng.choice([64, 100, 128, 200, 256, 384, 512])
            n = _log_int(rng, max(2000, 4 * m), 48000 if m <= 128 else 14000)
            ratio = rng.choice([0.03, 0.05, 0.1])
            kind, motifs, where = "ecg", 0, rng.choice(["host", "device", "oneshot"])
        else:
            m = rng.choice([64, 128, 200, 256, 400, 512, 777, 1024])
            ratio = rng.choice([0.01, 0.05, 0.05, 0.1, 0.2])
            hi = 100000 if ratio > 0.1 or m < 200 else 400000
            n = _log_int(rng, max(2000, 4 * m), hi)
            kind, motifs = "walk", rng.choice([0, 1]) if n >= 16 * m else 0
            where = rng.choice(["host", "device", "oneshot", "host", "device", "learned"])
        return dict(op="join", kind=kind, n=n, m=m, w=max(1, math.ceil(ratio * m)), motifs=motifs,
                    where=where)
    if op == "batch":
        return dict(op="batch", count=rng.randint(4, 32), lo=2000, hi=rng.choice([8192, 16384]))
    if op == "profile":
        m = rng.choice([32, 64, 128, 256, 500])
        return dict(op="profile", n=_log_int(rng, max(2000, 4 * m), 120000), m=m)
    if op == "pairs":
        m = rng.choice([64, 100, 128, 256, 512])
        return dict(op="pairs", n=_log_int(rng, 4000, 200000), m=m,
                    w=max(1, math.ceil(rng.choice([0.05, 0.1, 0.2]) * m)),
                    count=_log_int(rng, 200, 40000), precise=rng.choice([0, 1]),
                    where=rng.choice(["host", "device"]))
    return dict(op="train", rows=rng.choice([1000, 4096, 8192]), epochs=rng.randint(2, 12))


def _series(case, seed):
    synth = _synth()
    if case.get("kind", "walk") == "ecg":
        return synth.ecg_like(case["n"], seed)
    x = synth.random_walk(case["n"], seed)
    if case.get("motifs", 0):
        synth.plant_motifs(x, case["motifs"], case["m"], seed)
    return x


def _rows(case, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    d = _dtwj()
    x = rng.standard_normal((case["rows"], d.MLP_IN)).astype(np.float32)
    y = (0.5 * x[:, 0] + np.abs(x[:, 1]) + 0.1 * rng.standard_normal(case["rows"]))
    p = np.zeros(d.MLP_PARAMS, dtype=np.float32)  # W1, b1, W2, b2, w3, b3
    for at, count, fan in ((0, 8192, 64), (8320, 16384, 128), (24832, 128, 128)):
        a = math.sqrt(6.0 / fan)
        p[at:at + count] = rng.uniform(-a, a, count)
    return x, y.astype(np.float32), p


def _pair_lists(case, seed):
    rng = np.random.Generator(np.random.PCG64(seed + 1))
    s = case["n"] - case["m"] + 1
    return (rng.integers(0, s, case["count"]).astype(np.int64),
            rng.integers(0, s, case["count"]).astype(np.int64))


def prepare(case, seed):
    d = _dtwj()
    st = {"case": case}
    op = case["op"]
    if op == "train":
        st["x"], st["y"], st["p"] = _rows(case, seed)
        st["net"] = d.MLP(seed=1)
        return st
    if op == "batch":
        items = _synth().batch_workload(case["count"], seed, case["lo"], case["hi"])
        st["xs"] = [it["series"] for it in items]
        st["ms"] = [it["m"] for it in items]
        st["ws"] = [it["w"] for it in items]
        return st
    x = _series(case, seed)
    st["x"] = x
    if op == "join" and case["where"] != "oneshot":
        st["ctx"] = d.Context()
        if case["where"] == "device":
            st["dev"] = torch.from_numpy(x).cuda()
        if case["where"] == "learned":
            st["net"] = d.MLP.load_file(os.path.join(PKG, "tile_mlp_rw_m256.bin"))
            st["ctx"].set_model(st["net"])
    if op == "pairs":
        st["pi"], st["pj"] = _pair_lists(case, seed)
        if case["where"] == "device":
            st["dev"] = torch.from_numpy(x).cuda()
            st["dpi"] = torch.from_numpy(st["pi"]).cuda()
            st["dpj"] = torch.from_numpy(st["pj"]).cuda()
            st["out"] = torch.empty(case["count"], dtype=torch.float64, device="cuda")
    return st


def _pair_result(r):
    return {"i": r.i, "j": r.j, "dist": r.dist, "pairs": r.pairs}


def run(st):
    d = _dtwj()
    case = st["case"]
    op = case["op"]
    if op == "join":
        m, w = case["m"], case["w"]
        if case["where"] == "oneshot":
            return _pair_result(d.join(st["x"], m, w))
        if case["where"] == "device":
            return _pair_result(st["ctx"].join_device(st["dev"].data_ptr(), case["n"], m, w))
        flags = d.F_LEARNED if case["where"] == "learned" else 0
        return _pair_result(st["ctx"].join(st["x"], m, w, flags))
    if op == "batch":
        rs = d.join_batch(st["xs"], st["ms"], st["ws"])
        return {"i": np.array([r.i for r in rs]), "j": np.array([r.j for r in rs]),
                "dist": np.array([r.dist for r in rs])}
    if op == "profile":
        return d.matrix_profile(st["x"], case["m"])
    if op == "pairs":
        if case["where"] == "host":
            return d.pair_dtw(st["x"], case["m"], case["w"], st["pi"], st["pj"],
                              precise=bool(case["precise"]))
        p = ctypes.c_void_p
        rc = d.load().dtwj_pair_dtw_noalloc(
            p(st["dev"].data_ptr()), case["n"], case["m"], case["w"], p(st["dpi"].data_ptr()),
            p(st["dpj"].data_ptr()), case["count"], case["precise"], p(st["out"].data_ptr()),
            p(torch.cuda.current_stream().cuda_stream))
        if rc != d.OK:
            raise d.DtwjError(rc, "dtwj_pair_dtw_noalloc")
        return st["out"]
    # a fresh training run: weights set (which resets Adam), full-batch epochs
    st["net"].params = st["p"]
    loss = st["net"].train(st["x"], st["y"], epochs=case["epochs"], batch=case["rows"], lr=1e-3)
    return {"loss": loss, "params": st["net"].params}


def _pairs_of(n, m):
    k = n - 2 * m + 1  # windows that have a later partner at distance >= m
    return k * (k + 1) // 2


def work(case):
    """What a pass cannot do without.  A join or a profile reads the series
    once, and settles every candidate pair with one operation at the very
    least (one comparison of a bound); a pair list fills every band cell with
    a subtraction, a multiply-add and a minimum of three."""
    op = case["op"]
    if op == "join":
        return {"bytes": 8 * case["n"] + 32, "flops": _pairs_of(case["n"], case["m"])}
    if op == "batch":  # the expected length of a log-uniform draw, m = 128 on average
        mean = (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
        sq = (case["hi"] ** 2 - case["lo"] ** 2) / (2 * math.log(case["hi"] / case["lo"]))
        return {"bytes": 8 * mean * case["count"], "flops": case["count"] * 0.5 * sq}
    if op == "profile":
        s = case["n"] - case["m"] + 1
        return {"bytes": 8 * case["n"] + 16 * s, "flops": 4 * _pairs_of(case["n"], case["m"])}
    if op == "pairs":
        m, w = case["m"], min(case["w"], case["m"] - 1)
        cells = m * (2 * w + 1) - w * (w + 1)
        return {"bytes": 8 * case["n"] + 24 * case["count"], "flops": 5 * cells * case["count"]}
    flops = 6 * (64 * 128 + 128 * 128 + 128) * case["rows"] * case["epochs"]
    return {"bytes": (65 * 4 * case["rows"] + 4 * 24961), "flops": flops}


# ---- 64-bit results without this repository's code ----

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _windows(x, m, dev):
    """z-normalised windows [s][m] (population deviation), 64 bits."""
    w = torch.as_tensor(x, dtype=torch.float64, device=dev).unfold(0, m, 1)
    mu = w.mean(1, keepdim=True)
    z = w - mu
    return z / z.square().mean(1, keepdim=True).sqrt()


def _dtw_rows(q, t, w):
    """Banded DTW distance of many pairs at a time: q, t functions of a
    sample index returning the values of every pair."""
    m = q.m
    inf = math.inf
    prev = {}
    for r in range(m):
        cur = {}
        qr = q(r)
        for c in range(max(0, r - w), min(m, r + w + 1)):
            cost = (qr - t(c)).square()
            best = None
            for v in (prev.get(c - 1), prev.get(c), cur.get(c - 1)):
                if v is not None:
                    best = v if best is None else torch.minimum(best, v)
            if best is None:
                best = 0.0 if r == 0 and c == 0 else inf
            cur[c] = cost + best
        prev = cur
    return prev[m - 1].sqrt()


class _Columns:
    def __init__(self, m, get):
        self.m = m
        self.get = get

    def __call__(self, k):
        return self.get(k)


def _exact_join(x, m, w):
    dev = _device()
    s = len(x) - m + 1
    zt = _windows(x, m, dev).T.contiguous()  # [m][s]
    best = (math.inf, -1, -1)
    block = max(1, (1 << 23) // s)
    pad = torch.full((m, s + block), math.nan, dtype=torch.float64, device=dev)
    pad[:, :s] = zt
    for l0 in range(m, s, block):
        nl = min(block, s - l0)
        rows = s - l0
        q = _Columns(m, lambda k: zt[k, :rows].unsqueeze(0).expand(nl, rows))
        t = _Columns(m, lambda k: pad[k].unfold(0, rows, 1)[l0:l0 + nl])
        d = torch.nan_to_num(_dtw_rows(q, t, w), nan=math.inf)
        k = int(d.argmin())
        v = float(d.flatten()[k])
        i, lag = k % rows, l0 + k // rows
        best = min(best, (v, i, i + lag))
    return best


def exact(case, seed):
    op = case["op"]
    dev = _device()
    if op == "join":
        cells = _pairs_of(case["n"], case["m"]) * case["m"] * (2 * case["w"] + 1)
        if cells > 2e10:
            return None
        dist, i, j = _exact_join(_series(case, seed), case["m"], case["w"])
        return {"i": i, "j": j, "dist": dist, "pairs": _pairs_of(case["n"], case["m"])}
    if op == "batch":
        return None
    if op == "profile":
        m = case["m"]
        z = _windows(_series(case, seed), m, dev)
        s = z.shape[0]
        mp = torch.full((s,), math.inf, dtype=torch.float64, device=dev)
        mpi = torch.full((s,), -1, dtype=torch.int64, device=dev)
        cols = torch.arange(s, device=dev)
        for r0 in range(0, s, 2048):
            zr = z[r0:r0 + 2048]
            rows = torch.arange(r0, r0 + zr.shape[0], device=dev)
            corr = zr @ z.T
            corr.masked_fill_((cols - rows[:, None]).abs() < m, -math.inf)
            v, k = corr.max(1)
            ok = torch.isfinite(v)
            d = (zr - z[k]).square().sum(1).sqrt()
            mp[r0:r0 + 2048] = torch.where(ok, d, mp[r0:r0 + 2048])
            mpi[r0:r0 + 2048] = torch.where(ok, k, mpi[r0:r0 + 2048])
        return mp.cpu().numpy(), mpi.cpu().numpy()
    if op == "pairs":
        z = _windows(_series(case, seed), case["m"], dev)
        pi, pj = _pair_lists(case, seed)
        q = z[torch.from_numpy(pi).to(dev)].T.contiguous()
        t = z[torch.from_numpy(pj).to(dev)].T.contiguous()
        d = _dtw_rows(_Columns(case["m"], lambda k: q[k]), _Columns(case["m"], lambda k: t[k]),
                      min(case["w"], case["m"] - 1))
        return d.cpu().numpy() if case["where"] == "host" else d
    x, y, p = _rows(case, seed)
    x = torch.from_numpy(x).double().to(dev)
    y = torch.from_numpy(y).double().to(dev)
    p = torch.from_numpy(p).double().to(dev).requires_grad_(True)
    m1, m2 = torch.zeros_like(p), torch.zeros_like(p)
    loss = None
    for step in range(1, case["epochs"] + 1):
        w1, b1 = p[:8192].view(128, 64), p[8192:8320]
        w2, b2 = p[8320:24704].view(128, 128), p[24704:24832]
        w3, b3 = p[24832:24960], p[24960]
        h = torch.relu(torch.relu(x @ w1.T + b1) @ w2.T + b2)
        loss = (h @ w3 + b3 - y).square().mean()
        g, = torch.autograd.grad(loss, p)
        with torch.no_grad():
            m1.mul_(0.9).add_(g, alpha=0.1)
            m2.mul_(0.999).addcmul_(g, g, value=0.001)
            p -= 1e-3 * (m1 / (1 - 0.9 ** step)) / ((m2 / (1 - 0.999 ** step)).sqrt() + 1e-8)
    return {"loss": float(loss), "params": p.detach().cpu().numpy()}
