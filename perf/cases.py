"""The work whose speed is looked after: what programs have this framework do,
through its public entry points (p3arsec_gb300.Context, abi.Server).

A case is a dict of plain values.  Its "kind" names the entry point:

  host    Context.price_soa on host arrays -- the drop-in call and the CLI's
          ROI (num_runs passes between one copy in and one copy out);
  device  Context.price_soa on arrays resident on the GPU;
  f64     Context.price_soa_f64 on resident double arrays;
  books   Context.price_batch: many books of uneven size in one pool;
  serve   abi.Server: requests submitted together, then waited for;
  hjm     Context.price_swaptions: the swaptions application.

Books have the two field distributions of p3arsec_gb300.books: "plain" and
"tails".  Contexts are as bsg_create makes them (the drop-in CLIs never call
the autotuner).
"""
import math

import numpy as np
import torch

from p3arsec_gb300 import Context
from p3arsec_gb300 import books as B
from p3arsec_gb300 import swaptions as S
from p3arsec_gb300.abi import Server

DEV = "cuda:0"
MODES = ("fast", "sfu_ref", "libm_ref")
# floating operations of one evaluation of the formula (a division, square
# root, exp or log counted as one) and of one pair of normal variates (ten
# rounds of the generator left out)
FLOPS_OPTION = 62
FLOPS_PAIR = 40


def listed():
    return [
        # the smallest request of the serving trace, as one drop-in call
        {"name": "host_16", "kind": "host", "n": 16, "runs": 1, "mode": "fast", "dist": "plain", "pinned": False},
        # a book read from a file and priced once: pageable arrays, an odd size
        {"name": "host_1m", "kind": "host", "n": 1_000_003, "runs": 1, "mode": "fast", "dist": "plain", "pinned": False},
        # the benchmark's small input set as the CLI runs it: pinned arrays, NUM_RUNS = 100
        {"name": "roi_65536", "kind": "host", "n": 65_536, "runs": 100, "mode": "fast", "dist": "plain", "pinned": True},
        # the benchmark's 10M-option book, resident, NUM_RUNS = 100
        {"name": "map_10m", "kind": "device", "n": 10_000_000, "runs": 100, "mode": "fast", "dist": "plain", "offset": 0},
        # one shard of a resident book: any size, at an offset that is no multiple of a vector
        {"name": "map_shard", "kind": "device", "n": 1_250_001, "runs": 1, "mode": "fast", "dist": "plain", "offset": 3},
        # the precision sweep's book: the largest, 7.5 GB
        {"name": "map_2p28", "kind": "device", "n": 1 << 28, "runs": 1, "mode": "fast", "dist": "tails", "offset": 0},
        # the reference's own rounding for a large book
        {"name": "map_libm", "kind": "device", "n": 20_000_001, "runs": 1, "mode": "libm_ref", "dist": "tails", "offset": 0},
        # double prices
        {"name": "f64_4m", "kind": "f64", "n": 1 << 22, "runs": 1, "dist": "plain"},
        # 4,096 books of uneven size, about 45M options, one pass
        {"name": "books_4096", "kind": "books", "books": 4096, "max_len": 1 << 17, "runs": 1, "mode": "fast"},
        # a burst of requests of the serving trace's sizes
        {"name": "serve_64", "kind": "serve", "requests": 64, "min_n": 16, "max_n": 1 << 20},
        # the swaptions application's large input set
        {"name": "hjm_128x1m", "kind": "hjm", "swaptions": 128, "trials": 1_000_000, "steps": 11, "factors": 3},
        # and a small one
        {"name": "hjm_16x20k", "kind": "hjm", "swaptions": 16, "trials": 20_000, "steps": 11, "factors": 3},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    kind = rng.choice(["host", "device", "device", "f64", "books", "serve", "hjm"])
    dist = rng.choice(["plain", "tails"])
    if kind == "host":
        n = _log_int(rng, 1, 2_000_000)
        return {"kind": kind, "n": n, "runs": rng.choice([1, 1, 2, 10, 100]), "mode": rng.choice(MODES),
                "dist": dist, "pinned": rng.random() < 0.5}
    if kind == "device":
        n = _log_int(rng, 1000, 50_000_000)
        return {"kind": kind, "n": n, "runs": rng.choice([1, 1, 3, 10, 100]) if n <= 10_000_000 else 1,
                "mode": rng.choice(("fast", "fast") + MODES), "dist": dist, "offset": rng.choice([0, 0, 0, 1, 3, 4, 6])}
    if kind == "f64":
        return {"kind": kind, "n": _log_int(rng, 1000, 1 << 22), "runs": rng.choice([1, 1, 2]), "dist": dist}
    if kind == "books":
        return {"kind": kind, "books": _log_int(rng, 1, 4096), "max_len": _log_int(rng, 16, 1 << 17),
                "runs": rng.choice([1, 1, 2, 10]), "mode": rng.choice(("fast", "fast") + MODES)}
    if kind == "serve":
        return {"kind": kind, "requests": _log_int(rng, 1, 128), "min_n": 16, "max_n": _log_int(rng, 64, 1 << 18)}
    # the test suite's grids: the driver's 11 points and 3 factors, and others
    steps, factors = rng.choice([(11, 3), (11, 3), (11, 3), (7, 2), (12, 3), (20, 1), (25, 8), (32, 5)])
    return {"kind": kind, "swaptions": _log_int(rng, 1, 128),
            "trials": _log_int(rng, 1000, 1_000_000 if steps == 11 else 100_000), "steps": steps, "factors": factors}


# ------------------------------------------------------------------- inputs
def _log_uniform(lo, hi, count):
    """`count` sizes spread evenly over the logarithm of [lo, hi]."""
    q = (np.arange(count) + 0.5) / count
    return np.exp(math.log(lo) + q * math.log((hi + 1) / lo)).astype(np.int64)


def _book_segments(case, seed):
    """Books of lengths log-uniform in [1, max_len] in an order of the seed's
    own, each after a gap of 0 to 3 options: a pool's books start anywhere."""
    rng = np.random.default_rng(seed)
    lens = rng.permutation(_log_uniform(1, case["max_len"], case["books"]))
    gaps = rng.permutation(np.arange(case["books"]) % 4)
    ends = np.cumsum(lens + gaps)
    return [(int(e - n), int(n)) for e, n in zip(ends, lens)], int(ends[-1])


def _request_sizes(case, seed):
    """Request sizes log-uniform in [min_n, max_n], as the serving trace draws them."""
    sizes = _log_uniform(case["min_n"], case["max_n"], case["requests"])
    return [int(n) for n in np.random.default_rng(seed).permutation(sizes)]


def _swaptions(case, seed):
    if (case["steps"], case["factors"]) == (11, 3):
        return S.generate(case["swaptions"], seed)
    rng = np.random.default_rng(seed)
    n, nf = case["steps"], case["factors"]
    return [S.Swaption(strike=0.05 + 0.05 * rng.random(), years=0.5 * n, compounding=0.5 if i % 2 else 0.0,
                       payment_interval=0.5 if n >= 20 else 1.0, yield_curve=0.03 + 0.002 * np.arange(n),
                       factors=rng.uniform(-0.004, 0.012, (nf, n - 1)), seed=int(rng.integers(1, 1 << 31)))
            for i in range(case["swaptions"])]


def _host_arrays(arrays, pinned):
    if not pinned:
        return [np.ascontiguousarray(a.cpu().numpy()) for a in arrays], []
    keep = [a.cpu().pin_memory() for a in arrays]
    return [a.numpy() for a in keep], keep


def _inputs(case, seed):
    """The six arrays of a case's book (torch, on the GPU)."""
    kind = case["kind"]
    if kind == "books":
        n = _book_segments(case, seed)[1]
    elif kind == "serve":
        n = sum(_request_sizes(case, seed))
    else:
        n = case["n"] + case.get("offset", 0)
    return B.generate_device(n, seed, case.get("dist", "plain"), DEV)


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "hjm":
        st["swaptions"] = _swaptions(case, seed)
        st["ctx"] = Context(0, 1)
        return st
    arrays = _inputs(case, seed)
    n = arrays[0].numel()
    if kind == "host":
        st["arrays"], st["keep"] = _host_arrays(arrays, case["pinned"])
        st["prices"] = _host_arrays([torch.zeros(n)], case["pinned"])[0][0]
        st["ctx"] = Context(0, n)
    elif kind == "device":
        o = case["offset"]
        st["keep"] = arrays
        st["arrays"] = [a[o:] for a in arrays]
        st["prices"] = torch.zeros(n, dtype=torch.float32, device=DEV)[o:]
        st["ctx"] = Context(0, 1)
    elif kind == "f64":
        st["arrays"] = [a.double() for a in arrays[:5]] + [arrays[5]]
        st["prices"] = torch.zeros(n, dtype=torch.float64, device=DEV)
        st["ctx"] = Context(0, 1)
    elif kind == "books":
        st["segments"], st["pool_len"] = _book_segments(case, seed)
        st["arrays"] = arrays
        st["prices"] = torch.zeros(n, dtype=torch.float32, device=DEV)
        st["ctx"] = Context(0, 1)
    else:
        st["sizes"] = _request_sizes(case, seed)
        st["arrays"], st["keep"] = _host_arrays(arrays + [torch.zeros(n)], True)
        st["prices"] = st["arrays"].pop()
        st["server"] = Server(0, budget_bytes=1 << 30)
        for a in st["arrays"] + [st["prices"]]:
            st["server"].register(a)
    torch.cuda.synchronize()  # torch's fills are done before the context's stream reads them
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "hjm":
        return st["ctx"].price_swaptions(st["swaptions"], case["trials"])
    if kind == "host":
        return st["ctx"].price_soa(*st["arrays"], st["prices"], num_runs=case["runs"], mode=case["mode"])
    if kind == "device":
        return st["ctx"].price_soa(*st["arrays"], st["prices"], n=case["n"], num_runs=case["runs"],
                                   mode=case["mode"], device=True)
    if kind == "f64":
        return st["ctx"].price_soa_f64(*st["arrays"], st["prices"], n=case["n"], num_runs=case["runs"], device=True)
    if kind == "books":
        st["ctx"].price_batch(st["arrays"], st["prices"], st["pool_len"], st["segments"], num_runs=case["runs"],
                              mode=case["mode"])
        return st["prices"]
    srv, ids, at = st["server"], [], 0
    for n in st["sizes"]:
        ids.append(srv.submit(*[a[at:at + n] for a in st["arrays"]], st["prices"][at:at + n], n))
        at += n
    for i in ids:
        status, _ = srv.wait(i)
        if status != 0:
            raise RuntimeError("request %d ended with status %d" % (i, status))
    return st["prices"]


def work(case):
    kind = case["kind"]
    if kind == "hjm":
        # the variates up to maturity and the exponentials of the payments;
        # one year of maturity is one or two steps of the driver's grid
        if case["steps"] == 11:
            pairs, rates = 2, 3
        else:
            pairs, rates = case["factors"], 6
        per_path = pairs * FLOPS_PAIR + rates * (2 * case["factors"] + 2) + 3 * 12
        return {"bytes": case["swaptions"] * 16.0, "flops": float(case["swaptions"]) * case["trials"] * per_path}
    runs = case.get("runs", 1)
    if kind == "books":
        n = int(_log_uniform(1, case["max_len"], case["books"]).sum())
    elif kind == "serve":
        n = int(_log_uniform(case["min_n"], case["max_n"], case["requests"]).sum())
    else:
        n = case["n"]
    # every pass of num_runs reads the whole book and writes every price; a
    # book that crosses the host link does so once
    per = 52.0 if kind == "f64" else 28.0
    return {"bytes": per * n * (1 if kind == "host" else runs), "flops": float(FLOPS_OPTION) * n * runs}


# ------------------------------------------------------------ in 64 bits
def _cndf(x):
    """The polynomial of Abramowitz and Stegun 26.2.17 that the path evaluates."""
    k = 1.0 / (1.0 + 0.2316419 * x.abs())
    p = k * (0.319381530 + k * (-0.356563782 + k * (1.781477937 + k * (-1.821255978 + k * 1.330274429))))
    q = torch.exp(-0.5 * x * x) * 0.39894228040143270286 * p
    return torch.where(x < 0, q, 1.0 - q)


def _price64(s, k, r, v, t, ot):
    s, k, r, v, t = (a.double() for a in (s, k, r, v, t))
    den = v * torch.sqrt(t)
    d1 = ((r + 0.5 * v * v) * t + torch.log(s / k)) / den
    d2 = d1 - den
    fv = k * torch.exp(-r * t)
    call = s * _cndf(d1) - fv * _cndf(d2)
    put = fv * _cndf(-d2) - s * _cndf(-d1)
    return torch.where(ot == 0, call, put)


M32 = 0xFFFFFFFF


def _philox(seed, trial, pair):
    """Philox4x32-10 of the counter (trial, pair, 0) under the key seed, as four int64 tensors."""
    x = [trial & M32, (trial >> 32) & M32, torch.full_like(trial, pair), torch.zeros_like(trial)]
    k0, k1 = seed & M32, (seed >> 32) & M32
    for _ in range(10):
        p0, p1 = x[0] * 0xD2511F53, x[2] * 0xCD9E8D57
        x = [((p1 >> 32) & M32) ^ x[1] ^ k0, p1 & M32, ((p0 >> 32) & M32) ^ x[3] ^ k1, p0 & M32]
        k0, k1 = (k0 + 0x9E3779B9) & M32, (k1 + 0xBB67AE85) & M32
    return x


def _normals(seed, trial, count):
    out = []
    for j in range((count + 1) // 2):
        a, b, c, d = _philox(seed, trial, j)
        u1 = (2 * (((a >> 12) << 32) | b) + 1).double() * 2.0 ** -53
        u2 = (2 * (((c >> 12) << 32) | d) + 1).double() * 2.0 ** -53
        r = torch.sqrt(-2.0 * torch.log(u1))
        out += [r * torch.cos(2 * math.pi * u2), r * torch.sin(2 * math.pi * u2)]
    return out


def _swaption64(w, trials):
    """Price and standard error of one swaption: the HJM paths to maturity in 64 bits."""
    n, nf = w.n_steps, w.n_factors
    h = w.years / n
    strike = w.strike if w.compounding == 0 else math.log(1 + w.strike * w.compounding) / w.compounding
    freq, start, points = (int(x / h + 0.5) for x in (w.payment_interval, w.maturity, w.tenor))
    y, vol = w.yield_curve, w.factors
    fwd = [y[0]] + [(i + 1) * y[i] - i * y[i - 1] for i in range(1, n)]
    mu = [h * sum(vol[k][m] * (sum(vol[k][:m]) + 0.5 * vol[k][m]) for k in range(nf)) for m in range(n - 1)]
    trial = torch.arange(trials, device=DEV, dtype=torch.int64)
    z = _normals(w.seed, trial, start * nf)
    need = start + points - 1
    f = [torch.full((trials,), float(fwd[m]), dtype=torch.float64, device=DEV) for m in range(need + 1)]
    acc = torch.zeros_like(f[0])
    for i in range(start):
        acc += f[0]
        f = [f[m + 1] + mu[m] * h + math.sqrt(h) * sum(vol[k][m] * z[i * nf + k] for k in range(nf))
             for m in range(len(f) - 1)]
    fixed, accs = torch.zeros_like(acc), torch.zeros_like(acc)
    for m in range(points + 1):
        if m >= freq and m % freq == 0:
            pay = math.exp(strike * w.payment_interval) - (0 if m == points else 1)
            fixed += pay * torch.exp(-accs * h)
        if m < points:
            accs = accs + f[m]
    dp = torch.clamp(fixed - 1.0, min=0.0) * torch.exp(-acc * h)
    mean = dp.mean()
    err = torch.sqrt((dp - mean).square().sum() / (trials - 1.0)) / math.sqrt(trials)
    return float(mean), float(err)


def exact(case, seed):
    kind = case["kind"]
    if kind == "hjm":
        got = [_swaption64(w, case["trials"]) for w in _swaptions(case, seed)]
        return np.array([g[0] for g in got]), np.array([g[1] for g in got])
    arrays = _inputs(case, seed)
    o = case.get("offset", 0)
    n = arrays[0].numel() - o
    out = torch.zeros(n, dtype=torch.float64, device=DEV)
    spans = _book_segments(case, seed)[0] if kind == "books" else [(0, n)]
    if kind == "books":  # only the books are priced: the pool's gaps keep their zeros
        inside = torch.zeros(n + 1, dtype=torch.int32, device=DEV)
        inside[torch.tensor([a for a, _ in spans], device=DEV)] += 1
        ends = torch.tensor([a + m for a, m in spans], device=DEV)
        inside.index_add_(0, ends, torch.full_like(ends, -1, dtype=torch.int32))
        inside = inside.cumsum(0)[:n] > 0
    for a in range(0, n, 1 << 24):
        b = min(n, a + (1 << 24))
        p = _price64(*[x[o + a:o + b] for x in arrays])
        out[a:b] = torch.where(inside[a:b], p, 0.0) if kind == "books" else p
    return out.cpu().numpy() if kind in ("host", "serve") else out
