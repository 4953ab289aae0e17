"""What the speed of this framework is measured on: calls of its public entry
points over the range of sizes that its users run.

A case is a dict of plain values.  `kind` names the call:

  pi         pi(x) of one x with the library's y rule (the plain query, and
             what cpx-pi X prints)
  terms      pi_terms(x, y, c): every term of one x for a given alpha
  batch      pi_batch of n log-uniform x (one batched device pass, launched
             directly or as one CUDA graph, 64-bit or 128-bit kernels)
  gourdon    pi_gourdon(x)
  mu_lpf     mu and lpf of the odd numbers of a window, on the device
  count      the number of primes in a window
  pi_window  one window of a PiTable walk, on the device
  phi        phi(x, a)

Every state owns a context (stream, resident tables, work buffers) with the
committed tuning table, as a program that answers many such calls keeps one.
Results are whole numbers; those that can pass 64 bits come as two words.
"""
import math
import os
import random

import numpy as np
import torch

import cudapix_b200 as cpx

TUNING = os.path.join(os.path.dirname(os.path.abspath(cpx.__file__)), "tuning", "b200.json")


def listed():
    return [
        # the smallest call that takes the whole term pipeline: latency and launches
        {"name": "pi_1e8", "kind": "pi", "log10_x": 8.0},
        # the reference's own configuration: x = 1e12, y = 1e5, c = 6
        {"name": "terms_1e12", "kind": "terms", "log10_x": 12.0, "alpha": 10, "c": 6},
        # one ordinary and one large query in 64 bits, and one in 128 bits (x > 2^64)
        {"name": "pi_1e15", "kind": "pi", "log10_x": 15.0},
        {"name": "pi_1e17", "kind": "pi", "log10_x": 17.0},
        {"name": "pi_2e19", "kind": "pi", "log10_x": 19.275},
        # the benchmark's batch
        {"name": "batch_4096", "kind": "batch", "n": 4096, "lo": 9.0, "hi": 14.0, "graph": False, "wide": False},
        # a smaller batch of larger queries, as one CUDA graph
        {"name": "batch_1024_graph", "kind": "batch", "n": 1024, "lo": 10.0, "hi": 15.0, "graph": True,
         "wide": False},
        # the second decomposition
        {"name": "gourdon_1e15", "kind": "gourdon", "log10_x": 15.0},
        # the sieves and tables that programs call on their own
        {"name": "mu_lpf_1e12", "kind": "mu_lpf", "log10_lo": 12.0, "odd": 30_000_000},
        {"name": "count_1e12", "kind": "count", "log10_lo": 12.0, "span": 10_000_000_000},
        {"name": "pi_window_1e10", "kind": "pi_window", "log10_lo": 10.0, "span": 100_000_000},
        {"name": "phi_1e10", "kind": "phi", "log10_x": 10.0, "a": 100},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pi", "terms", "batch", "gourdon", "mu_lpf", "count", "pi_window", "phi"])
    c = {"kind": kind}
    if kind == "pi":
        c["log10_x"] = round(rng.uniform(6.0, 18.5), 4)
    elif kind == "terms":
        c.update(log10_x=round(rng.uniform(9.0, 16.5), 4), alpha=rng.randint(2, 32), c=rng.choice([4, 5, 6, 7]))
    elif kind == "batch":
        lo = rng.uniform(7.0, 11.0)
        hi = rng.uniform(lo + 1.0, 14.0)
        c.update(n=_log(rng, 3, 4096), lo=round(lo, 3), hi=round(hi, 3), graph=rng.random() < 0.4,
                 wide=rng.random() < 0.15)
    elif kind == "gourdon":
        c["log10_x"] = round(rng.uniform(8.0, 16.5), 4)
    elif kind == "mu_lpf":
        c.update(log10_lo=round(rng.uniform(3.0, 13.0), 4), odd=_log(rng, 5_000, 30_000_000))
    elif kind == "count":
        c.update(log10_lo=round(rng.uniform(3.0, 13.0), 4), span=_log(rng, 10_000, 10_000_000_000))
    elif kind == "pi_window":
        c.update(log10_lo=round(rng.uniform(3.0, 11.0), 4), span=2 * _log(rng, 5_000, 50_000_000))
    else:
        c.update(log10_x=round(rng.uniform(5.0, 10.0), 4), a=_log(rng, 2, 2000))
    return c


# ------------------------------------------------------------------ inputs

def _inputs(case, seed):
    """The call's arguments, from the seed alone: x or lo within 2% of the
    case's size, the x of a batch log-uniform in its range."""
    rng = random.Random(int(seed) * 1_000_003 + 17)
    kind = case["kind"]
    if kind == "batch":
        e = np.random.default_rng(int(seed)).uniform(case["lo"], case["hi"], case["n"])
        return {"xs": [int(10.0**v) for v in e]}
    near = 1.0 + rng.uniform(-0.02, 0.0)
    if kind in ("mu_lpf", "count", "pi_window"):
        lo = int(10.0 ** case["log10_lo"] * near)
        if kind != "count":
            lo &= ~1
        if kind == "mu_lpf":
            return {"lo": lo, "hi": lo + 2 * case["odd"]}
        return {"lo": lo, "hi": lo + case["span"]}
    x = int(10.0 ** case["log10_x"] * near)
    a = {"x": x}
    if kind == "terms":
        a["y"] = cpx.default_y(x, case["alpha"])
    return a


def _context():
    ctx = cpx.Context(0)
    ctx.tune_load(TUNING)
    return ctx


def prepare(case, seed):
    a = _inputs(case, seed)
    ctx = _context()
    if case["kind"] == "pi_window":
        a["table"] = cpx.PiTable(a["lo"], 0, case["span"], ctx=ctx)
    if case["kind"] == "phi":
        a["phi"] = cpx.Phi(0, ctx=ctx)
    a.update(kind=case["kind"], ctx=ctx, case=case)
    return a


# --------------------------------------------------------------------- run

def _words(v):
    """A whole number of up to 128 bits (two's complement) as two 64-bit words."""
    v &= (1 << 128) - 1
    return np.array([v & 0xFFFFFFFFFFFFFFFF, v >> 64], dtype=np.uint64).view(np.int64)


class _Device:
    """A device array of the library as torch sees it, without a copy; the
    array lives as long as the tensor."""

    def __init__(self, arr, typestr):
        self.arr = arr
        self.__cuda_array_interface__ = {"shape": (arr.n,), "typestr": typestr, "data": (arr.ptr, False),
                                         "version": 3}


def _tensor(arr, typestr):
    return torch.as_tensor(_Device(arr, typestr), device="cuda")


_TERMS = ("P2", "ordinary", "trivial", "easy", "hard", "pi_y", "pi", "y")
_GOURDON = ("A", "B", "C", "D", "phi0", "sigma", "pi", "y")


def run(s):
    kind, ctx, case = s["kind"], s["ctx"], s["case"]
    if kind == "pi":
        return cpx.pi(s["x"], ctx=ctx)
    if kind == "terms":
        t = cpx.pi_terms(s["x"], s["y"], case["c"], ctx=ctx)
        return {k: _words(t[k]) for k in _TERMS}
    if kind == "batch":
        return np.array(cpx.pi_batch(s["xs"], wide=case["wide"], graph=case["graph"], ctx=ctx), dtype=np.int64)
    if kind == "gourdon":
        t = cpx.pi_gourdon(s["x"], ctx=ctx)
        return {k: _words(t[k]) for k in _GOURDON}
    if kind == "mu_lpf":
        mu, lpf = cpx.gen_d_mu_lpf(s["lo"], s["hi"], ctx=ctx)
        return {"mu": _tensor(mu, "|i1"), "lpf": _tensor(lpf, "<i8")}
    if kind == "count":
        return cpx.count_primes(s["lo"], s["hi"], ctx=ctx)
    if kind == "pi_window":
        t = s["table"].getCurrent()
        return {"table": _tensor(t, "<i4"), "pi_base": s["table"].get_pi_base()}
    return s["phi"].phi_std(s["x"], case["a"])


# -------------------------------------------------------------------- work

def _pi_ops(x):
    """Operations of pi(x) by Deleglise-Rivat, in the order of its bound
    x^(2/3) / log^2 x (leaves and sieve)."""
    return x ** (2.0 / 3.0) / math.log(x) ** 2


def work(case):
    """Inputs read once, outputs written once; flops are whole-number operations."""
    kind = case["kind"]
    if kind == "batch":
        # mean of x^(2/3) / log^2 x over the batch, in the exponent
        es = np.linspace(case["lo"], case["hi"], 257)
        ops = float(np.mean([_pi_ops(10.0**e) for e in es])) * case["n"]
        return {"bytes": 32 * case["n"], "flops": ops}
    if kind == "mu_lpf":
        return {"bytes": 9 * case["odd"], "flops": 3 * case["odd"]}
    if kind == "count":
        return {"bytes": 24, "flops": case["span"]}
    if kind == "pi_window":
        # the window's odd numbers, and the count of the primes below it
        return {"bytes": 2 * case["span"], "flops": case["span"] + 10.0 ** case["log10_lo"]}
    x = 10.0 ** case["log10_x"]
    if kind == "phi":
        # crossings of the odd numbers up to x by p_2 .. p_a
        return {"bytes": 16, "flops": x / 2 * max(0.5, math.log(math.log(6.0 + case["a"] * math.log(2.0 + case["a"]))))}
    return {"bytes": 64, "flops": _pi_ops(x)}


# ------------------------------------------------------------------- exact

def _small_primes(n):
    s = np.ones(n + 1, dtype=bool)
    s[:2] = False
    for p in range(2, math.isqrt(n) + 1):
        if s[p]:
            s[p * p::p] = False
    return np.nonzero(s)[0]


def _sieve(lo, hi, ps):
    """True where no p of ps divides n (n = p itself included), n in [lo, hi)."""
    s = np.ones(hi - lo, dtype=bool)
    for p in ps:
        s[-lo % p::p] = False
    return s


def _primes(lo, hi):
    ps = [int(p) for p in _small_primes(math.isqrt(hi) + 1)]
    s = _sieve(lo, hi, ps)
    for p in ps:
        if lo <= p < hi:
            s[p - lo] = True
    s[:max(0, 2 - lo)] = False
    return np.nonzero(s)[0].astype(np.int64) + lo


def _mu_lpf(lo, hi):
    """mu and lpf of the odd n in [lo, hi) (lpf(1) = 2^32 - 1)."""
    n = np.arange(lo + 1, hi, 2, dtype=np.int64)
    rest, mu, lpf = n.copy(), np.ones(n.size, dtype=np.int8), np.zeros(n.size, dtype=np.int64)
    for p in _small_primes(math.isqrt(hi) + 1)[1:]:
        p = int(p)
        i0 = (-(lo + 1) * pow(2, -1, p)) % p  # the first i with p | lo + 1 + 2 i
        at = slice(i0, None, p)
        lpf[at] = np.where(lpf[at] == 0, p, lpf[at])
        mu[at] = -mu[at]
        rest[at] //= p
        p2 = p * p
        if p2 < hi:
            mu[(-(lo + 1) * pow(2, -1, p2)) % p2::p2] = 0
            k = p2
            while k < hi:  # divide out the higher powers too
                rest[(-(lo + 1) * pow(2, -1, k)) % k::k] //= p
                k *= p
    big = rest > 1
    mu[big] = -mu[big]
    lpf = np.where(lpf == 0, n, lpf)
    lpf[n == 1] = 0xFFFFFFFF
    return mu, lpf


def exact(case, seed):
    a, kind = _inputs(case, seed), case["kind"]
    if kind == "pi" and a["x"] <= 200_000_000:
        return int(_small_primes(a["x"]).size)
    if kind == "count" and a["hi"] - a["lo"] <= 20_000_000 and a["hi"] <= 2 * 10**12:
        return int(_primes(a["lo"], a["hi"]).size)
    if kind == "pi_window" and a["hi"] <= 100_000_000:
        # table[k] = pi(lo + 2k - 1) - pi(lo - 1), k < span / 2 + 2
        ps = _small_primes(a["hi"] + 4)
        base = int(np.searchsorted(ps, a["lo"]))
        n = a["lo"] - 1 + 2 * np.arange(case["span"] // 2 + 2, dtype=np.int64)
        return {"table": np.searchsorted(ps, n, side="right") - base, "pi_base": base}
    if kind == "mu_lpf" and case["odd"] <= 1_000_000 and a["hi"] <= 10**11:
        mu, lpf = _mu_lpf(a["lo"], a["hi"])
        return {"mu": mu, "lpf": lpf}
    if kind == "phi" and a["x"] <= 50_000_000:
        s = _sieve(1, a["x"] + 1, [int(p) for p in _small_primes(20_000)[:case["a"]]])
        return int(s.sum())
    return None
