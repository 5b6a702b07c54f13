"""The work that programs ask of the engine, as measurable cases.

Each case is one pass of a program written with the array front end. Except for the interactive
one, the program's flush is compiled once (Runtime.take, NativeExecutor.compile) and executed on
every pass, as a program that repeats an array expression does; inputs and outputs stay in the
engine's device buffers. The kinds, and what each stands for:

  interactive   a short expression on a small array, recorded, flushed and read back on every pass:
                the latency a user of the prompt or of a scalar loop sees
  chain         r = sum(sqrt(a*a + b*b) * exp(-c)), float64: one fused map with a full reduction
  blackscholes  European call prices, float64 (about 44 bytecodes), ending in the mean price
  heat          ten Jacobi steps of the 5-point heat stencil over shifted views, float32, each with
                the largest change as its convergence measure
  life          ten generations of the game of life on an integer grid (8 shifted views, comparisons
                and logic): integer and boolean work on odd, small grids
  batch         independent float32 systems of uneven length in one flush, grouped launches: a
                12-operation chain kept per system, its sum and its maximum
  scan          cumsum(2x + 1) of a long vector
  summed_area   the summed-area table of an image: cumulative sums along both axes
  transpose     C = A + B^T: a map that reads one operand through a transposed view
  softmax       row-wise softmax: a maximum and a sum over the contiguous axis, and maps between
  standardise   columns to zero mean and unit variance: sums over the outermost axis, broadcasts
  montecarlo    pi from uniform random points: the counter-based generator and a full reduction

Sizes come from the benchmark's workloads where it has them (2^20 chain, 10M options, 4096^2 heat,
5e7 scan, 8192^2 transpose, lengths 256..65536 for the batch) and are generic otherwise.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import bohrium_b200 as bh
from bohrium_b200 import workloads as W
from bohrium_b200.array import accumulate, binary, random_sample

_EPS = 1e-5  # variance floor of the standardisation


def listed():
    return [
        # the smallest call: latency of recording, flushing and reading one number back
        {"name": "interactive_f64_1000", "kind": "interactive", "dtype": "float64", "n": 1000},
        # the plain fused block of ordinary size
        {"name": "chain_f64_1m", "kind": "chain", "dtype": "float64", "n": 1 << 20},
        # map-heavy pricing at full size
        {"name": "blackscholes_f64_10m", "kind": "blackscholes", "dtype": "float64", "n": 10_000_000},
        # stencil at full size
        {"name": "heat_f32_4096", "kind": "heat", "dtype": "float32", "rows": 4096, "cols": 4096},
        # a small odd integer grid: ten dependent launches that each take microseconds
        {"name": "life_i32_517x1023", "kind": "life", "dtype": "int32", "rows": 517, "cols": 1023},
        # many small independent blocks in one flush
        {"name": "batch_f32_20", "kind": "batch", "dtype": "float32", "systems": 20, "lengths": 3},
        # a long prefix sum
        {"name": "scan_f64_50m", "kind": "scan", "dtype": "float64", "n": 50_000_000},
        # accumulation along each axis of an image with odd rows
        {"name": "summed_area_f32_4000x4099", "kind": "summed_area", "dtype": "float32", "rows": 4000, "cols": 4099},
        # a transposed operand whose rows are not a multiple of 16 bytes
        {"name": "transpose_f32_8191x6001", "kind": "transpose", "dtype": "float32", "rows": 8191, "cols": 6001},
        # many rows of ordinary length
        {"name": "softmax_f32_20000x1500", "kind": "softmax", "dtype": "float32", "rows": 20000, "cols": 1500},
        # a tall table of few columns
        {"name": "standardise_f64_500003x50", "kind": "standardise", "dtype": "float64", "rows": 500003, "cols": 50},
        # random numbers, no input
        {"name": "montecarlo_f64_50m", "kind": "montecarlo", "dtype": "float64", "n": 50_000_000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["interactive", "chain", "blackscholes", "heat", "life", "batch", "scan", "summed_area",
                       "transpose", "softmax", "standardise", "montecarlo"])
    real = rng.choice(["float32", "float64"])
    if kind == "interactive":
        return {"kind": kind, "dtype": real, "n": _log_int(rng, 100, 100_000)}
    if kind == "chain":
        return {"kind": kind, "dtype": real, "n": _log_int(rng, 10_000, 30_000_000)}
    if kind == "blackscholes":
        return {"kind": kind, "dtype": "float64", "n": _log_int(rng, 100_000, 10_000_000)}
    if kind == "heat":
        return {"kind": kind, "dtype": real, "rows": _log_int(rng, 200, 4096), "cols": _log_int(rng, 200, 2048)}
    if kind == "life":
        return {"kind": kind, "dtype": rng.choice(["int32", "int64"]), "rows": _log_int(rng, 100, 3000),
                "cols": _log_int(rng, 100, 3000)}
    if kind == "batch":
        return {"kind": kind, "dtype": "float32", "systems": rng.randint(4, 20), "lengths": rng.randrange(1 << 16)}
    if kind == "scan":
        return {"kind": kind, "dtype": rng.choice(["float32", "float64", "int64"]), "n": _log_int(rng, 10_000, 50_000_000)}
    if kind == "summed_area":
        return {"kind": kind, "dtype": rng.choice(["float32", "float64", "int32"]), "rows": _log_int(rng, 100, 5000),
                "cols": _log_int(rng, 100, 4000)}
    if kind == "transpose":
        even = rng.random() < 0.5  # rows of a multiple of 16 bytes, or as they come
        r, c = _log_int(rng, 200, 8192), _log_int(rng, 200, 4096)
        return {"kind": kind, "dtype": rng.choice(["float32", "float64", "int32"]),
                "rows": r // 4 * 4 if even else r, "cols": c // 4 * 4 if even else c}
    if kind == "softmax":
        return {"kind": kind, "dtype": real, "rows": _log_int(rng, 50, 20000), "cols": _log_int(rng, 10, 1500)}
    if kind == "standardise":
        return {"kind": kind, "dtype": real, "rows": _log_int(rng, 1000, 500_000), "cols": _log_int(rng, 4, 50)}
    return {"kind": kind, "dtype": real, "n": _log_int(rng, 10_000, 50_000_000)}


# ------------------------------------------------------------------------------------- inputs
def _torch_dtype(case):
    return getattr(torch, case["dtype"])


def _inputs(case, seed, device="cuda"):
    """The case's input tensors, from the seed alone."""
    g = torch.Generator(device=device)
    g.manual_seed(int(seed) * 7919 + 17)
    dt = _torch_dtype(case)

    def uniform(shape, lo=0.0, hi=1.0):
        return torch.rand(shape, generator=g, device=device, dtype=dt) * (hi - lo) + lo

    def ints(shape, lo, hi):
        return torch.randint(lo, hi, shape, generator=g, device=device, dtype=dt)

    kind = case["kind"]
    if kind in ("interactive", "chain"):
        return [uniform((case["n"],)) for _ in range(3)]
    if kind == "blackscholes":
        n = (case["n"],)
        return [uniform(n, 5.0, 30.0), uniform(n, 1.0, 100.0), uniform(n, 0.25, 10.0)]
    if kind == "heat":
        x = torch.ones((case["rows"], case["cols"]), device=device, dtype=dt)
        x[1:-1, 1:-1] = uniform((case["rows"] - 2, case["cols"] - 2))
        return [x]
    if kind == "life":
        return [ints((case["rows"], case["cols"]), 0, 2)]
    if kind == "batch":
        return [uniform((int(n),)) for n in _lengths(case)]
    if kind == "scan":
        return [ints((case["n"],), -50, 50) if dt == torch.int64 else uniform((case["n"],))]
    if kind == "transpose":
        shapes = [(case["rows"], case["cols"]), (case["cols"], case["rows"])]
        return [ints(s, -1000, 1000) if dt == torch.int32 else uniform(s) for s in shapes]
    if kind == "summed_area":
        s = (case["rows"], case["cols"])
        return [ints(s, 0, 256) if dt == torch.int32 else uniform(s)]
    if kind == "softmax":
        return [torch.randn((case["rows"], case["cols"]), generator=g, device=device, dtype=dt) * 3.0]
    if kind == "standardise":
        return [torch.randn((case["rows"], case["cols"]), generator=g, device=device, dtype=dt) * 2.0 + 5.0]
    return []


def _lengths(case):
    return W.batching_lengths(case["systems"], 256, 65536, case["lengths"])


# ------------------------------------------------------------------------------------ programs
def _life_step(src, dst):
    c = src[1:-1, 1:-1]
    n = (src[:-2, :-2] + src[:-2, 1:-1] + src[:-2, 2:] + src[1:-1, :-2] + src[1:-1, 2:] +
         src[2:, :-2] + src[2:, 1:-1] + src[2:, 2:])
    dst[1:-1, 1:-1] = (n == 3) | ((n == 2) & (c == 1))


def _program(rt, case, seed, x):
    """Record the case's program on the arrays `x`; returns the arrays it leaves."""
    kind = case["kind"]
    if kind in ("interactive", "chain"):
        return [W.plain_chain(rt, *x)]
    if kind == "blackscholes":
        return [W.black_scholes_iteration(rt, *x, 1)]
    if kind in ("heat", "life"):
        # Ten steps from the given grid: the first leaves it untouched, the others alternate
        # between two grids that already hold the boundary.
        grid, ping, pong = x
        src, dst, deltas = grid, ping, []
        for _ in range(10):
            if kind == "heat":
                deltas.append(W.heat_step(src, dst))
            else:
                _life_step(src, dst)
            src, dst = dst, (pong if dst is ping else ping)
        return [src] + deltas
    if kind == "batch":
        outs = []
        for a in x:
            y = W.batching_chain(a)
            outs += [y, y.sum(), y.max()]
        return outs
    if kind == "scan":
        return [accumulate("ADD_ACCUMULATE", x[0] * 2 + 1, 0)]
    if kind == "summed_area":
        return [x[0].cumsum(0).cumsum(1)]
    if kind == "transpose":
        return [x[0] + x[1].T]
    if kind == "softmax":
        rows = case["rows"]
        m = x[0].max(1)
        e = bh.exp(x[0] - m.reshape(rows, 1))
        return [e / e.sum(1).reshape(rows, 1)]
    if kind == "standardise":
        n = float(case["rows"])
        mean = x[0].sum(0) / n
        d = x[0] - mean
        var = (d * d).sum(0) / n
        return [d / bh.sqrt(var + _EPS), mean, var]
    n, dt = case["n"], np.dtype(case["dtype"]).type
    px = random_sample(rt, (n,), start=0, key=1000 + int(seed), dtype=dt)
    py = random_sample(rt, (n,), start=1 << 40, key=1000 + int(seed), dtype=dt)
    inside = (px * px + py * py <= dt(1)).astype(dt)
    return [inside.sum() * dt(4) / dt(n)]


# ------------------------------------------------------------------------------------- running
_runtimes = {}


def _runtime(mode):
    """One engine per batching mode for the whole program, with its instruction queue."""
    if mode not in _runtimes:
        ex = bh.NativeExecutor()
        ex.message("CUDA: batch " + mode)
        _runtimes[mode] = bh.Runtime(ex)
    return _runtimes[mode]


class _Device:
    def __init__(self, pointer, shape, dtype):
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": np.dtype(dtype).str, "data": (pointer, False),
                                         "version": 3}


def _device_tensor(rt, a):
    """The engine's device buffer of array `a` (a whole base) as a tensor."""
    p = rt.ex.lib.bhb_data_get(rt.ex.rt, a.base.handle, 0, 1, 0)
    if not p:
        raise RuntimeError("bhb_data_get: " + (rt.ex.lib.bhb_last_error() or b"").decode())
    return torch.as_tensor(_Device(p, a.shape, a.dtype), device="cuda")


def prepare(case, seed):
    rt = _runtime("grouped" if case["kind"] == "batch" else "off")
    rt.flush()  # arrays that earlier programs dropped are freed
    given = _inputs(case, seed)
    arrays = []
    for t in given + (given * 2 if case["kind"] in ("heat", "life") else []):
        a = bh.empty(rt, tuple(t.shape), np.dtype(case["dtype"]))
        _device_tensor(rt, a).copy_(t)
        arrays.append(a)
    torch.cuda.synchronize()
    state = {"kind": case["kind"], "rt": rt, "arrays": arrays}
    if case["kind"] == "interactive":
        return state
    outs = _program(rt, case, seed, arrays)
    state["ir"] = rt.ex.compile(rt.take())
    state["outs"] = outs
    state["tensors"] = [_device_tensor(rt, o) for o in outs]
    return state


def run(state):
    if state["kind"] == "interactive":
        return _program(state["rt"], {"kind": "interactive"}, 0, state["arrays"])[0].numpy()
    state["ir"].execute()
    return state["tensors"]


# -------------------------------------------------------------------------------------- checks
def _philox(start, key, n, device):
    """Philox2x32-10 (Salmon et al., 2011) of the 64-bit counters start .. start+n-1, as the two
    32-bit words of each result."""
    mask = 0xFFFFFFFF
    ctr = torch.arange(n, device=device, dtype=torch.int64) + start
    lo, hi, k = ctr & mask, (ctr >> 32) & mask, key & mask
    m_hi, m_lo = 0xD256D193 >> 16, 0xD256D193 & 0xFFFF
    for r in range(10):
        # 32 x 32 -> 64 bit product in two halves that stay below 2^63
        a, b = lo * m_lo, lo * m_hi
        low = (a + ((b & 0xFFFF) << 16))
        p_hi, p_lo = (b >> 16) + (low >> 32), low & mask
        lo, hi = p_hi ^ k ^ hi, p_lo
        k = (k + 0x9E3779B9) & mask
    return lo, hi


def exact(case, seed):
    x = [t.double() if t.is_floating_point() else t for t in _inputs(case, seed)]
    kind = case["kind"]
    if kind in ("interactive", "chain"):
        r = (torch.sqrt(x[0] * x[0] + x[1] * x[1]) * torch.exp(-x[2])).sum()
        return r.cpu().numpy() if kind == "interactive" else [r]
    if kind == "blackscholes":
        S, K, T = x
        r, vol = 0.02, 0.3

        def cnd(v):
            v = v * (1.0 / math.sqrt(2.0))
            a = v.abs()
            t = 1.0 / (1.0 + W.AS_P * a)
            c = W.AS_A
            poly = ((((c[4] * t + c[3]) * t + c[2]) * t + c[1]) * t + c[0]) * t
            return 0.5 * (1.0 + torch.sign(v) * (1.0 - poly * torch.exp(-(a * a))))

        T = T * 1.01
        sq = torch.sqrt(T)
        d1 = (torch.log(S / K) + (r + 0.5 * vol * vol) * T) / (vol * sq)
        d2 = d1 - vol * sq
        return [(S * cnd(d1) - K * torch.exp(-r * T) * cnd(d2)).mean()]
    if kind == "heat":
        g, deltas, f = x[0].clone(), [], float(np.float32(0.2))
        for _ in range(10):
            c = g[1:-1, 1:-1]
            w = (c + g[:-2, 1:-1] + g[2:, 1:-1] + g[1:-1, :-2] + g[1:-1, 2:]) * f
            deltas.append((w - c).abs().max())
            g = g.clone()
            g[1:-1, 1:-1] = w
        return [g] + deltas
    if kind == "life":
        g = x[0].clone()
        for _ in range(10):
            c = g[1:-1, 1:-1]
            n = (g[:-2, :-2] + g[:-2, 1:-1] + g[:-2, 2:] + g[1:-1, :-2] + g[1:-1, 2:] +
                 g[2:, :-2] + g[2:, 1:-1] + g[2:, 2:])
            w = ((n == 3) | ((n == 2) & (c == 1))).to(g.dtype)
            g = g.clone()
            g[1:-1, 1:-1] = w
        return [g]
    if kind == "batch":
        outs = []
        for a in x:
            y = a * 1.5 + 0.25
            y = torch.sqrt((y * y - 0.125).abs())
            y = torch.maximum(torch.exp(-y) * 2.0, torch.full_like(y, 0.5)) + a
            y = y * 0.75 - 0.0625
            outs += [y, y.sum(), y.max()]
        return outs
    if kind == "scan":
        return [torch.cumsum(x[0] * 2 + 1, 0)]
    if kind == "summed_area":
        return [torch.cumsum(torch.cumsum(x[0], 0, dtype=x[0].dtype), 1, dtype=x[0].dtype)]
    if kind == "transpose":
        return [x[0] + x[1].T]
    if kind == "softmax":
        return [torch.softmax(x[0], 1)]
    if kind == "standardise":
        mean = x[0].mean(0)
        d = x[0] - mean
        var = (d * d).mean(0)
        return [d / torch.sqrt(var + _EPS), mean, var]
    # float32 points and sums round: the count near the circle has no 64-bit counterpart there
    if case["dtype"] != "float64":
        return None
    n, inside = case["n"], 0
    for at in range(0, n, 1 << 24):
        m = min(1 << 24, n - at)
        p = []
        for start in (0, 1 << 40):
            lo, hi = _philox(start + at, 1000 + int(seed), m, "cuda")
            p.append((hi.double() * 4294967296.0 + lo.double()) / float(np.iinfo(np.uint64).max))
        inside += int((p[0] * p[0] + p[1] * p[1] <= 1.0).sum())
    return [torch.tensor(4.0 * inside / n, dtype=torch.float64)]


# ---------------------------------------------------------------------------------------- work
def work(case):
    kind, size = case["kind"], np.dtype(case["dtype"]).itemsize
    n = case.get("n", case.get("rows", 0) * case.get("cols", 0))
    if kind in ("interactive", "chain"):
        return {"bytes": 3 * size * n + size, "flops": 8 * n}
    if kind == "blackscholes":
        return {"bytes": 3 * size * n + size, "flops": 70 * n}
    if kind in ("heat", "life"):
        # every step reads its grid and writes the next one's interior
        inner = (case["rows"] - 2) * (case["cols"] - 2)
        return {"bytes": 10 * size * (n + inner), "flops": 10 * inner * (8 if kind == "heat" else 12)}
    if kind == "batch":
        n = int(_lengths(case).sum())
        return {"bytes": 2 * size * n + 2 * size * case["systems"], "flops": 14 * n}
    if kind == "scan":
        return {"bytes": 2 * size * n, "flops": 3 * n}
    if kind == "summed_area":
        return {"bytes": 2 * size * n, "flops": 2 * n}
    if kind == "transpose":
        return {"bytes": 3 * size * n, "flops": n}
    if kind == "softmax":
        return {"bytes": 2 * size * n, "flops": 5 * n}
    if kind == "standardise":
        return {"bytes": 2 * size * n + 2 * size * case["cols"], "flops": 6 * n}
    return {"bytes": size, "flops": 90 * n}  # two generated numbers a point: integer multiplies and xors
