"""What the performance of this package is judged by: batched tridiagonal solves
through the public Python entry points, over the sizes, types and layouts that
they are used with.

A case is one call on device-resident inputs: a solver (`kind`), the system
size `n`, the batch `m`, the type and, where the solver has one, its option
(`rest` = CR-to-PCR switch level, `g` = Thomas chains).  The inputs are the
distributions of the benchmark: strictly diagonally dominant systems, weakly
dominant ones for the large systems, ADI lines for the ragged batches.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import tridiagonalsolvers_gb300 as tg
from tridiagonalsolvers_gb300 import ragged

#: kind -> what one pass calls
POW2 = ("cr", "crNBC", "pcr", "crpcr", "pcrGauss")
BYTES = {"f32": 4, "f64": 8}


def listed():
    return [
        # The smallest call of a loop over small batches: 5 MB, latency and launches count.
        dict(name="cr_f32_512x512", kind="cr", dtype="f32", n=512, m=512),
        # The headline: a large batch of short systems, one call of the drop-in CR.
        dict(name="cr_f32_256x65536", kind="cr", dtype="f32", n=256, m=65536),
        # The second large batch of the benchmark, with the solver that does the most arithmetic.
        dict(name="pcr_f32_1024x16384", kind="pcr", dtype="f32", n=1024, m=16384),
        # The hybrid on longer systems, a batch that is no round number.
        dict(name="crpcr_f32_2048x6001", kind="crpcr", dtype="f32", n=2048, m=6001, rest=64),
        # PCR-then-Thomas with the reference driver's 64 chains, at the longest systems it takes.
        dict(name="pcrGauss_f32_4096x2048", kind="pcrGauss", dtype="f32", n=4096, m=2048, g=64),
        # The reference's USE_DOUBLE build of its CR, on the second large batch.
        dict(name="cr_f64_1024x16384", kind="cr", dtype="f64", n=1024, m=16384),
        # The any-size solver on short systems that are no power of two, rows off the 16-byte grid.
        dict(name="solve_f32_250x65536", kind="solve", dtype="f32", n=250, m=65536),
        # The same in double precision, ordinary sizes.
        dict(name="solve_f64_1000x4096", kind="solve", dtype="f64", n=1000, m=4096),
        # Few long lines, each contiguous, odd sizes (spline fits, 1-D implicit steps).
        dict(name="large_f32_100001x257", kind="large", dtype="f32", n=100001, m=257, layout="contiguous"),
        # The large interleaved batch of the benchmark, plain ...
        dict(name="large_f32_inter_65536x1024", kind="large", dtype="f32", n=65536, m=1024, layout="interleaved"),
        # ... and refined to 1e-10.
        dict(name="refine_inter_65536x1024", kind="refine", dtype="f32", n=65536, m=1024, layout="interleaved"),
        # The ragged batch of ADI lines, refined in one launch (the largest case).
        dict(name="ragged_refine_100000", kind="ragged_refine", dtype="f32", lo=32, hi=8192, m=100000),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["cr", "crNBC", "pcr", "crpcr", "pcrGauss", "solve", "solve", "large", "large", "refine", "ragged",
                       "ragged_refine"])
    dtype = "f64" if kind in POW2 + ("solve", "large") and rng.random() < 0.3 else "f32"
    if kind in POW2:
        n = 1 << rng.randint(5, 12)
        if kind == "crNBC" and dtype == "f64":
            n = min(n, 2048)
        most = (1 << 24) if dtype == "f32" else (1 << 22)
        case = dict(kind=kind, dtype=dtype, n=n, m=_log_int(rng, max(1, (1 << 15) // n), most // n))
        if kind == "crpcr":
            case["rest"] = 1 << rng.randint(1, n.bit_length() - 2)
        if kind == "pcrGauss":
            case["g"] = 1 << rng.randint(3, n.bit_length() - 1)
    elif kind == "solve":
        n = _log_int(rng, 20, 8000 if dtype == "f32" else 4000)
        case = dict(kind=kind, dtype=dtype, n=n, m=_log_int(rng, max(1, (1 << 15) // n), (1 << 24) // n))
    elif kind == "large":
        n = _log_int(rng, 9000, 1000000)
        most = (1 << 25) if dtype == "f32" else (1 << 24)
        case = dict(kind=kind, dtype=dtype, n=n, m=_log_int(rng, 1, max(1, min(2048, most // n))),
                    layout=rng.choice(["contiguous", "interleaved"]))
    elif kind == "refine":
        layout = rng.choice(["contiguous", "interleaved"])
        n = _log_int(rng, 64, 8000) if layout == "contiguous" else _log_int(rng, 9000, 100000)
        case = dict(kind=kind, dtype=dtype, n=n, m=_log_int(rng, max(1, (1 << 16) // n), (1 << 24) // n), layout=layout)
    else:
        lo, hi = _log_int(rng, 32, 300), _log_int(rng, 600, 12000)
        case = dict(kind=kind, dtype=dtype, lo=lo, hi=hi, m=_log_int(rng, 100, 20000))
    return case


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _uniform(g, shape, lo, hi):
    return torch.empty(shape, dtype=torch.float32, device="cuda").uniform_(lo, hi, generator=g)


def _offsets(case):
    """Sizes log-uniform in [lo, hi], concatenated; the same ones for every seed."""
    rng = np.random.default_rng([case["m"], case["lo"], case["hi"]])
    sizes = np.exp(rng.uniform(np.log(case["lo"]), np.log(case["hi"] + 1), case["m"])).astype(np.int64)
    off = np.zeros(case["m"] + 1, np.int64)
    np.cumsum(np.clip(sizes, case["lo"], case["hi"]), out=off[1:])
    return off


def _inputs(case, seed):
    g = _gen(seed)
    if "lo" in case:  # ADI lines: a = c = -r, b = 1 + 2r, one r a system
        off = _offsets(case)
        rows, need = int(off[-1]), ragged.padded(off[-1])
        at = torch.from_numpy(off).cuda()
        r = _uniform(g, (case["m"],), 0.1, 10.0).repeat_interleave(at[1:] - at[:-1], output_size=rows)
        a = torch.zeros(need, dtype=torch.float32, device="cuda")
        b = torch.ones(need, dtype=torch.float32, device="cuda")
        a[:rows] = -r
        b[:rows] += 2 * r
        del r
        c, d = a.clone(), _uniform(g, (need,), -1.0, 1.0)
        a[at[:-1]] = 0
        c[at[1:] - 1] = 0
        return off, (a, b, c, d)
    n, m = case["n"], case["m"]
    inter = case.get("layout") == "interleaved"
    shape = (n, m) if inter else (m, n)
    weak = case["kind"] == "large" or inter  # the large systems of the benchmark are weakly dominant
    a, c = _uniform(g, shape, -1.0, 1.0), _uniform(g, shape, -1.0, 1.0)
    if inter:
        a[0], c[-1] = 0, 0
    else:
        a[:, 0], c[:, -1] = 0, 0
    b = a.abs() + c.abs() + (_uniform(g, shape, 0.01, 0.1) if weak else _uniform(g, shape, 1.0, 2.0))
    d = _uniform(g, shape, -1.0, 1.0)
    if case["dtype"] == "f64":
        a, b, c, d = (t.double() for t in (a, b, c, d))
    if "layout" in case:
        a, b, c, d = (t.reshape(-1) for t in (a, b, c, d))
    return None, (a, b, c, d)


def prepare(case, seed):
    off, ins = _inputs(case, seed)
    state = {"case": case, "in": ins}
    if case["kind"] == "ragged":
        state["plan"] = ragged.RaggedPlan(off)
    elif case["kind"] == "ragged_refine":
        state["refiner"] = ragged.RaggedRefiner(ragged.RaggedPlan(off, refine=True), *ins, sweeps=1)
    return state


def run(state):
    case, ins = state["case"], state["in"]
    kind = case["kind"]
    if kind == "crpcr":
        return tg.crpcr(*ins, case["rest"])
    if kind == "pcrGauss":
        return tg.pcrGauss(*ins, case["g"])
    if kind == "large":
        return tg.solve_large(*ins, case["n"], case["m"], layout=case["layout"])
    if kind == "refine":  # the residual it also returns is rounding noise near 1e-13
        x, sweeps, _ = tg.refine(*ins, case["n"], case["m"], layout=case["layout"], tol=1e-10)
        return {"x": x, "sweeps": sweeps}
    if kind == "ragged":
        return state["plan"].solve(*ins)
    if kind == "ragged_refine":
        state["refiner"].launch()
        return state["refiner"].x
    return getattr(tg, kind)(*ins)


def _rows(case):
    if "lo" not in case:
        return case["n"] * case["m"]
    # the mean of a log-uniform size
    return int(case["m"] * (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"]))


def work(case):
    """a, b, c, d read once and x written once (in FP64 by the refinements); the
    operations of the shortest elimination: 8 forward and back a row, for a
    refinement two of them and two residuals of 14 in extended precision."""
    size = BYTES[case["dtype"]]
    refined = "refine" in case["kind"]
    per_row = 4 * size + (8 if refined else size)
    return {"bytes": per_row * _rows(case), "flops": (2 * 8 + 2 * 14 if refined else 8) * _rows(case)}


def _solve64(a, b, c, d, stride, longest):
    """Parallel cyclic reduction in FP64 on all rows at once: neighbours `stride`
    rows apart; the couplings across systems are zero, so they drop out."""
    a, b, c, d = (t.reshape(-1).double() for t in (a, b, c, d))
    # each row divided by its diagonal: x = d - a x[-1] - c x[+1]
    a, c, d = a / b, c / b, d / b
    del b
    step, dist = stride, 1

    def left(t):
        return torch.cat([torch.zeros(step, dtype=t.dtype, device=t.device), t[:-step]])

    def right(t):
        return torch.cat([t[step:], torch.zeros(step, dtype=t.dtype, device=t.device)])

    while dist < longest and step < a.numel():
        inv = 1.0 / (1.0 - a * left(c) - c * right(a))
        d = (d - a * left(d) - c * right(d)) * inv
        a, c = -a * left(a) * inv, -c * right(c) * inv
        step, dist = 2 * step, 2 * dist
    return d


def exact(case, seed):
    off, ins = _inputs(case, seed)
    if off is not None:
        rows = int(off[-1])
        x = _solve64(*(t[:rows] for t in ins), 1, int(np.diff(off).max()))
        pad = torch.zeros(ragged.padded(rows) - rows, dtype=torch.float64, device=x.device)
        return torch.cat([x, pad])
    inter = case.get("layout") == "interleaved"
    x = _solve64(*ins, case["m"] if inter else 1, case["n"]).reshape(ins[0].shape)
    return {"x": x, "sweeps": None} if case["kind"] == "refine" else x
