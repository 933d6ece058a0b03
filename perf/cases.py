"""The work this library is measured on, through its public entry points.

A case is a plain dict.  `kind` says which entry point a pass goes through:

  range   Engine.run_job: device sieve of a p range, walk, output rule
  list    Engine.check_primes: a host list of primes, as the app.h plugin feeds it
  raw     Engine.check_primes_raw: the same, every candidate, as the appcu.h layer
  device  Engine.check_primes_device: a list of primes already on the GPU
  input   Engine.run_job with an input sieve file as the output rule
  sieve   Engine.sieve_range: the count and sum of a range's primes
  batch   Engine.run_batch: many mixed jobs in one call
  serve   Server.submit / wait: the same kind of jobs through the serving loop

and the other values say the job: primes from plo (plus a seeded offset below
`spread`), k in [kmin, kmax], n in [nmin, nmin + nw), side (+1, -1, 2: twin), and
`width` of the p range or `count` primes or jobs.
"""
import math
import random
import sys
import tempfile
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "psieve-cuda_gb300"))

import ppsgpu  # noqa: E402

LARGE_N = dict(plo=42 * 10**12, spread=10**11, kmin=1201, kmax=9999, nmin=2000000, nw=1000000, side=1)
RIESEL62 = dict(plo=(1 << 62) - (1 << 34), spread=(1 << 34) - (1 << 31), kmin=3, kmax=9999, nmin=100000,
                nw=900000, side=-1)
SMALL_PROTH = dict(plo=10**12, spread=10**10, kmin=1201, kmax=9999, nmin=2000, nw=1000, side=1)
MID_RIESEL = dict(plo=3 * 10**12, spread=10**11, kmin=3, kmax=9999, nmin=65537, nw=131071, side=-1)

# 512-job mixes run for seconds; the sizes here keep their distribution and cut the p widths.
MIX_SCALE_P = 0.25


def listed():
    return [
        # the smallest call: the appcu.h layer asked for a few primes' candidates (latency)
        dict(name="raw_1000", kind="raw", count=1000, plo=6 * 10**11, spread=10**10, kmin=1201, kmax=9999,
             nmin=2000000, nw=1000000, side=1),
        # a whole small search, short n range (sieve, set-up and launches): pps/app.c's small Proth range
        dict(name="small_proth_full", kind="range", width=2 * 10**8, **SMALL_PROTH),
        # the reference's own 2e6-wide test slice of the large-n range: few primes, a million n
        dict(name="large_n_2e6", kind="range", width=2 * 10**6, **LARGE_N),
        # one batch of the app.h plugin: 2,048 primes per SM in pageable host memory
        dict(name="plugin_batch", kind="list", count=2048 * 152, **LARGE_N),
        # an odd number of primes already on the GPU, steps shorter than 32, mid n range
        dict(name="device_mid_riesel", kind="device", count=1000003, **MID_RIESEL),
        # the primes of a p slice, as a run is checked: the count=, sum= line of the reference
        dict(name="sieve_slice", kind="sieve", width=(1 << 31) + 1, **LARGE_N),
        # production: a p slice of the large-n Proth search
        dict(name="large_n_slice", kind="range", width=1 << 30, **LARGE_N),
        # production: a p slice near 2^62, Riesel side
        dict(name="riesel62_slice", kind="range", width=1 << 30, **RIESEL62),
        # production: both sides of twin candidates from one walk
        dict(name="twin_slice", kind="range", width=1 << 28, **dict(LARGE_N, kmin=3, side=2)),
        # the second pass over a range with candidates left in a sieve file
        dict(name="input_slice", kind="input", width=1 << 28, records=200000, **LARGE_N),
        # many uneven jobs in one call
        dict(name="batch_96", kind="batch", count=96, plo=0, spread=0),
        # the same kind of jobs through the serving loop, all submitted at once
        dict(name="serve_24", kind="serve", count=24, plo=0, spread=0),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Jobs of the mixed-job distribution's ranges (p from 1e12 up, where every
    k and n width below is accepted), through every entry point."""
    kind = rng.choice(["range", "range", "list", "raw", "device", "input", "sieve", "batch", "serve"])
    if kind == "batch":
        return dict(kind=kind, count=_log_uniform(rng, 2, 96), plo=0, spread=0)
    if kind == "serve":
        return dict(kind=kind, count=_log_uniform(rng, 1, 24), plo=0, spread=0)
    plo = _log_uniform(rng, 10**12, 1 << 61)
    kmin = 2 * rng.randrange(1, 2500) + 1
    case = dict(kind=kind, plo=plo, spread=10**9, kmin=kmin, kmax=kmin + 2 * (_log_uniform(rng, 100, 5000) // 2),
                nmin=rng.randrange(1000, 2000001), nw=_log_uniform(rng, 1000, 1000000), side=rng.choice([1, -1, 2]))
    if kind == "sieve":
        return dict(case, width=_log_uniform(rng, 10**6, 1 << 31))
    if kind == "input":
        case["records"] = _log_uniform(rng, 1000, 200000)
        case["side"] = rng.choice([1, -1])
    # at most half the largest listed case's walk steps (3.4e7 primes x 31,250)
    most = min(3 * 10**7, int(5e11 / (case["nw"] / 24)))
    count = _log_uniform(rng, 500, most)
    if kind in ("range", "input"):
        return dict(case, width=max(20000, int(count * math.log(plo))))
    if case["side"] == 2:
        case["side"] = rng.choice([1, -1])  # list entry points: one side
    return dict(case, count=min(count, 2000000))


# A program holds one engine (and one server) for its life and passes jobs to it.
_held = {}


def _engine():
    if "engine" not in _held:
        _held["engine"] = ppsgpu.Engine(0)
    return _held["engine"]


def _server():
    if "server" not in _held:
        _held["server"] = ppsgpu.Server(0)
    return _held["server"]


def _plo(case, seed):
    return case["plo"] + 2 * random.Random(seed * 7 + 1).randrange(max(case["spread"] // 2, 1))


def _job(case, plo, width):
    return ppsgpu.normalize(pmin=plo, pmax=plo + width, kmin=case["kmin"], kmax=case["kmax"], nmin=case["nmin"],
                            nmax=case["nmin"] + case["nw"], sign=case["side"])


def _mixed(case, seed):
    return ppsgpu.mixed_jobs(seed=seed + 1, count=case["count"], scale_p=MIX_SCALE_P)[0]


def _primes(case, plo):
    """`count` consecutive primes from plo, and the end of their range."""
    width = int(case["count"] * math.log(plo) * 1.1) + 20000
    primes, n, _ = _engine().sieve_range(plo, plo + width, want_primes=True, cap=2 * case["count"] + 4096)
    primes = primes[: case["count"]].copy()
    return primes, int(primes[-1]) + 2 - plo


def _sieve_file(case, seed):
    """A NewPGen file of `records` seeded (k, n) of the job's ranges."""
    rng = np.random.default_rng(seed)
    n = case["records"]
    ks = rng.integers(case["kmin"] // 2, case["kmax"] // 2 + 1, size=n) * 2 + 1
    ns = rng.integers(case["nmin"], case["nmin"] + case["nw"], size=n)
    # the two ends keep the scanned extents the job's
    ks[0], ns[0], ks[1], ns[1] = case["kmin"] | 1, case["nmin"], case["kmax"] | 1, case["nmin"] + case["nw"] - 1
    order = np.lexsort((ks, ns))
    head = "%d:P:1:2:%d" % (case["plo"], case["side"])
    with tempfile.NamedTemporaryFile("w", suffix=".txt", delete=False) as f:
        f.write(head + "\n")
        f.writelines("%d %d\n" % (ks[i], ns[i]) for i in order)
    return f.name


def _room(case):
    """Lines a pass of the case may give: four times the expected candidates."""
    if case["kind"] in ("batch", "serve"):
        return 1 << 16
    if case["kind"] == "sieve":
        return 0
    primes = case.get("count") or case["width"] / math.log(case["plo"])
    expect = (case["kmax"] - case["kmin"] + 2) / 2 * case["nw"] * primes / case["plo"]
    return int(4 * expect) + 256


def prepare(case, seed):
    kind, room = case["kind"], _room(case)
    if kind in ("batch", "serve"):
        on = _engine() if kind == "batch" else _server()
        return {"kind": kind, "room": room, "on": on, "jobs": _mixed(case, seed)}
    plo = _plo(case, seed)
    state = {"kind": kind, "room": room, "on": _engine() if kind != "input" else None}
    if kind == "sieve":
        return dict(state, lo=plo, hi=plo + case["width"])
    if kind == "range":
        return dict(state, job=_job(case, plo, case["width"]))
    if kind == "input":
        path = _sieve_file(case, seed)
        inp = ppsgpu.InputFile(path, pmin=plo, pmax=plo + case["width"], sign=case["side"])
        Path(path).unlink()
        # the file belongs to an engine of its own: its table is made at the engine's first call
        eng = ppsgpu.Engine(0)
        eng.set_input(inp)
        return dict(state, on=eng, job=ppsgpu.normalize(**inp.spec))
    primes, width = _primes(case, plo)
    state["job"] = _job(case, plo, width)
    if kind == "device":
        dev = torch.from_numpy(primes.view(np.int64)).cuda()
        torch.cuda.synchronize()
        return dict(state, primes=dev)
    return dict(state, primes=primes)


def _rows(arr, fields, room):
    """Records as whole numbers, their count first, in a buffer of `room` rows."""
    out = np.zeros((room, len(fields)), dtype=np.int64)
    n = min(len(arr), room)
    for i, f in enumerate(fields):
        out[:n, i] = arr[f][:n]
    return [len(arr), out]


_LINE = ("p", "k", "n", "c")


def run(state):
    """One call, and what it gives.  The list entry points name primes by value
    or index, so the list itself (the state's own buffer) goes with them."""
    kind, on, room = state["kind"], state["on"], state["room"]
    if kind in ("range", "input"):
        fac, st = on.run_job(state["job"])
        return _rows(fac, _LINE, room) + [int(st.primes), int(st.prime_sum) & (2**63 - 1)]
    if kind == "list":
        fac, st = on.check_primes(state["job"], state["primes"])
        return _rows(fac, _LINE, room) + [int(st.primes), state["primes"].view(np.int64)]
    if kind == "raw":
        hits = on.check_primes_raw(state["job"], state["primes"])
        return _rows(hits, ("p", "k", "n", "idx"), room) + [state["primes"].view(np.int64)]
    if kind == "device":
        fac, st = on.check_primes_device(state["job"], state["primes"].data_ptr(), state["primes"].numel())
        return _rows(fac, _LINE, room) + [int(st.primes), state["primes"]]
    if kind == "sieve":
        _, count, total = on.sieve_range(state["lo"], state["hi"])
        return [int(count), int(total) & (2**63 - 1)]
    if kind == "batch":
        per, _ = on.run_batch(state["jobs"])
        count, total = on.batch_job_primes(len(state["jobs"]))
        return _rows(np.concatenate(per), _LINE, room) + [count.view(np.int64), total.view(np.int64)]
    ids = [on.submit(j) for j in state["jobs"]]
    per = [on.wait(i) for i in ids]
    return _rows(np.concatenate([f for f, _ in per]), _LINE, room) + [
        np.array([[r.primes, r.prime_sum & (2**63 - 1), r.factors] for _, r in per], dtype=np.int64)]


def _job_work(plo, width, nw, step, nbytes):
    """One job: its primes' n ranges at the fewest multiplies of the recurrence
    k <- k 2^-step mod p (three 32-bit multiplies a step of a prime)."""
    primes = width / math.log(max(plo, 3))
    return nbytes(primes), 2 * 3 * primes * math.ceil(nw / step)


def work(case):
    kind = case["kind"]
    if kind in ("batch", "serve"):
        total = [0.0, 0.0]
        for j in _mixed(case, 0):
            w = _job_work(j.pmin, j.pmax - j.pmin, j.nmax - j.nmin, j.step, lambda n: 64)
            total = [total[0] + w[0], total[1] + w[1]]
        return {"bytes": total[0], "flops": total[1]}
    plo = case["plo"]
    width = case.get("width") or case["count"] * math.log(plo)
    if kind == "sieve":
        # each odd candidate is struck once per sieving prime dividing it
        return {"bytes": 16, "flops": width / 2 * math.log(math.log(math.sqrt(plo)))}
    job = _job(dict(case, side=case["side"]), plo, int(width) + 2)
    nbytes = (lambda n: 64) if kind in ("range", "input") else (lambda n: 8 * n)
    b, f = _job_work(plo, width, case["nw"], job.step, nbytes)
    return {"bytes": b + 16 * case.get("records", 0), "flops": f}


def exact(case, seed):
    """Every output is a whole number: they are compared as they are."""
    return None
