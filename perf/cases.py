"""The work a user of the skycube engine has it do, as cases that can be timed.

A case names a kind of call ("use"), a dataset shape and distribution, and the
options of the call. The kinds are the ways a program reaches the engine:

  cube     skycube of a dataset resident on the device, its per-cuboid skyline
           ids read on the device (offsets and ids)
  query    skyline of one subspace of a resident dataset, ids on the device
  plain    the per-cuboid SDSC form of the suite, extended skylines included
  plan     replay of a planned (captured) skycube of a resident dataset
  host     host rows in, every cuboid's ids out on the host: upload, skycube,
           one host list per cuboid
  bitmaps  per-point dominated-subspace bitmaps, on the host
  serve    a burst of skyline and skycube requests on host rows through the
           serving loop, every answer's ids on the host

Inputs are drawn on the GPU from the seed with the distributions of
skycube_gb300.datagen. All outputs are ids, offsets or bitmaps: whole numbers.
How many ids there are follows from the data, so the program keeps an id table
with room for them (zeros behind the last id) and gathers each answer there.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "skycube-templates_gb300"))

import skycube_gb300 as sk  # noqa: E402

KINDS = ("uniform", "correlated", "anticorrelated", "ties", "correlated_q")


def listed():
    return [
        # The smallest calls: an interactive skyline query and a whole skycube
        # of a few thousand rows, where latency and launches count.
        {"name": "query-1k-4", "use": "query", "kind": "uniform", "n": 1000, "d": 4, "subspace": 0b1011},
        {"name": "cube-5k-8", "use": "cube", "kind": "correlated", "n": 5003, "d": 8, "max_d": 0},
        # The suite's own schedule on its small benchmark shape (63 cuboids,
        # one launch sequence each).
        {"name": "plain-100k-6", "use": "plain", "kind": "uniform", "n": 100000, "d": 6, "max_d": 0},
        # A new table from host memory, all 31 skylines back in host memory.
        {"name": "host-250k-5", "use": "host", "kind": "uniform", "n": 250007, "d": 5, "max_d": 0},
        # A skyline query on a large table: 7 of 12 attributes.
        {"name": "query-1m-12", "use": "query", "kind": "uniform", "n": 1000000, "d": 12,
         "subspace": 0b010110111010},
        # The headline: every cuboid of a million anticorrelated points.
        {"name": "cube-1m-10", "use": "cube", "kind": "anticorrelated", "n": 1000000, "d": 10, "max_d": 0},
        # Integer-valued data with many duplicates and ties.
        {"name": "ties-581k-10", "use": "cube", "kind": "ties", "n": 581012, "d": 10, "max_d": 0},
        # Quantised correlated data, cuboids of at most 6 attributes, replayed
        # as a plan (9,949 cuboids).
        {"name": "plan-566k-15-m6", "use": "plan", "kind": "correlated_q", "n": 566268, "d": 15, "max_d": 6},
        # Capped skycubes of 16 attributes, the shape of the suite's published
        # sweeps; the second is the largest case.
        {"name": "cube-500k-16-m4", "use": "cube", "kind": "anticorrelated", "n": 500000, "d": 16, "max_d": 4},
        {"name": "cube-500k-16-m6", "use": "cube", "kind": "anticorrelated", "n": 500000, "d": 16, "max_d": 6},
        # Per-point dominated-subspace bitmaps, as the suite's MDMC keeps them.
        {"name": "bitmaps-200k-9", "use": "bitmaps", "kind": "uniform", "n": 200003, "d": 9, "max_d": 0},
        # A burst of mixed requests on a running server.
        {"name": "serve-burst", "use": "serve", "queries": 8, "n_max": 200000, "mix": 5},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same uses: n log-uniform from 1,000 up to a
    million (less where a larger one would cost more than the largest listed
    case), 4 to 16 attributes."""
    use = rng.choice(("query", "query", "cube", "cube", "capped", "capped", "plain", "plan",
                      "host", "bitmaps", "serve"))
    kind = rng.choice(KINDS)
    if use == "query":
        d = rng.randint(4, 16)
        n = _log_int(rng, 1000, 1000000 if d <= 12 else 500000)
        while True:
            s = rng.randrange(1, 1 << d)
            if bin(s).count("1") >= 2:
                return {"use": use, "kind": kind, "n": n, "d": d, "subspace": s}
    if use == "cube":
        return {"use": use, "kind": kind, "n": _log_int(rng, 1000, 1000000), "d": rng.randint(4, 10),
                "max_d": 0}
    if use == "capped":
        return {"use": "cube", "kind": kind, "n": _log_int(rng, 5000, 400000), "d": rng.randint(9, 16),
                "max_d": rng.randint(2, 6)}
    if use == "plain":
        return {"use": use, "kind": kind, "n": _log_int(rng, 1000, 150000), "d": rng.randint(4, 6),
                "max_d": 0}
    if use == "plan":
        if rng.random() < 0.5:
            return {"use": use, "kind": kind, "n": _log_int(rng, 1000, 500000), "d": rng.randint(4, 9),
                    "max_d": 0}
        return {"use": use, "kind": "correlated_q", "n": _log_int(rng, 10000, 600000),
                "d": rng.randint(11, 15), "max_d": rng.randint(3, 6)}
    if use == "host":
        return {"use": use, "kind": kind, "n": _log_int(rng, 1000, 1000000), "d": rng.randint(4, 6),
                "max_d": 0}
    if use == "bitmaps":
        return {"use": use, "kind": kind, "n": _log_int(rng, 1000, 300000), "d": rng.randint(6, 11),
                "max_d": 0}
    return {"use": use, "queries": rng.randint(4, 12), "n_max": _log_int(rng, 20000, 300000),
            "mix": rng.randrange(1 << 20)}


# ---------------------------------------------------------------------------
# Inputs

def _anticorrelated(g, n, d):
    out, filled = [], 0
    while filled < n:
        m = max(1024, int((n - filled) * 1.5))
        v = torch.randn(m, 1, generator=g, device="cuda", dtype=torch.float64) * 0.05 + 0.5
        x = torch.rand(m, d, generator=g, device="cuda", dtype=torch.float64)
        x += v - x.mean(dim=1, keepdim=True)
        x = x[((x >= 0) & (x <= 1)).all(dim=1)][: n - filled]
        out.append(x)
        filled += x.shape[0]
    return torch.cat(out)


def _correlated(g, n, d):
    v = (torch.randn(n, 1, generator=g, device="cuda", dtype=torch.float64) * 0.25 + 0.5).clamp(0, 1)
    e = torch.randn(n, d, generator=g, device="cuda", dtype=torch.float64) * 0.05
    return (v + e).clamp(0, 1)


def _points(kind, n, d, seed):
    """(n, d) float32 points on the GPU (the distributions of datagen)."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    if kind == "uniform":
        x = torch.rand(n, d, generator=g, device="cuda", dtype=torch.float64)
    elif kind == "anticorrelated":
        x = _anticorrelated(g, n, d)
    elif kind == "correlated":
        x = _correlated(g, n, d)
    elif kind == "ties":
        c = (n * 4) // 10
        x = torch.cat([torch.rand(n - c, d, generator=g, device="cuda", dtype=torch.float64),
                       _correlated(g, c, d)])
        x = torch.floor(256.0 * x[torch.randperm(n, generator=g, device="cuda")])
    else:
        x = torch.round(_correlated(g, n, d) / (0.1 / d)) * (0.1 / d)
    return x.to(torch.float32).contiguous()


def _requests(case):
    """The burst's requests: half skyline queries on a random subspace, half
    skycubes (every cuboid up to 6 attributes, else capped at 2)."""
    rng = random.Random(case["mix"])
    got = []
    for i in range(case["queries"]):
        d = rng.randint(4, 12)
        q = {"kind": rng.choice(KINDS[:3]), "n": _log_int(rng, 1000, case["n_max"]), "d": d}
        if i % 2:
            q.update(max_d=d if d <= 6 else 2, subspace=0)
        else:
            q.update(max_d=0, subspace=rng.randrange(3, 1 << d) | 3)
        got.append(q)
    return got


_ctx = None


def _context():
    """One engine context per process, as a user's program keeps it."""
    global _ctx
    if _ctx is None:
        _ctx = sk.Context(0)
    return _ctx


def _cuboids(d, max_d):
    return [c for c in range(1, 1 << d)
            if max_d <= 0 or bin(c).count("1") <= max_d or c == (1 << d) - 1]


def _room(kind, n, d, max_d):
    """Ids to keep room for: with (ln n)^j / j! summed over j < k as the
    skyline of k independent attributes, the points clipped to the best value
    on all k of correlated data, and the distribution's factor on top."""
    total = n
    for k in range(1, (max_d if 0 < max_d < d else d) + 1):
        e = sum(math.log(n) ** j / math.factorial(j) for j in range(k))
        if kind == "anticorrelated":
            e *= 2.0 * 1.35 ** max(0, k - 4)
        elif kind != "uniform":
            e += 0.04 * n / 2 ** k
        total += math.comb(d, k) * min(n, 1.5 * e + 64)
    return int(total)


# ---------------------------------------------------------------------------

def prepare(case, seed):
    ctx = _context()
    use = case["use"]
    if use == "serve":
        reqs = _requests(case)
        for i, q in enumerate(reqs):
            q["x"] = _points(q["kind"], q["n"], q["d"], int(seed) * 1000 + i).cpu().numpy()
            q["cuboids"] = [q["subspace"]] if q["subspace"] else _cuboids(q["d"], q["max_d"])
            room = q["n"] if q["subspace"] else _room(q["kind"], q["n"], q["d"], q["max_d"])
            q["ids"] = np.zeros(room, np.int32)
        return {"use": use, "server": sk.Server(ctx, slots=4), "requests": reqs}
    n, d = case["n"], case["d"]
    x = _points(case["kind"], n, d, seed)
    state = {"use": use, "ctx": ctx, "d": d}
    room = n if use == "query" else _room(case["kind"], n, d, case["max_d"])
    if use == "host":
        state["x"] = x.cpu().numpy()
        state["cuboids"] = _cuboids(d, 0)
        state["ids"] = np.zeros(room, np.int32)
        return state
    if use == "bitmaps":
        state["bits"] = np.zeros((n, max(1, (1 << d) // 32)), np.uint32)
        state["points"] = np.zeros(n, np.uint32)
    else:
        state["ids"] = torch.zeros(room, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()  # the engine reads x on a stream of its own
    state["ds"] = sk.Dataset(ctx, device_ptr=x.data_ptr(), n=n, d=d)
    if use == "query":
        state["opts"] = {"subspace": case["subspace"]}
    elif use == "plain":
        state["opts"] = {"algo": "sdsc", "mode": "plain", "max_d": case["max_d"], "want_extended": True}
    elif use == "bitmaps":
        state["opts"] = {"max_d": case["max_d"], "want_bitmaps": True}
    else:
        state["opts"] = {"max_d": case["max_d"]}
    if use == "plan":
        state["plan"] = sk.Plan(ctx, state["ds"], **state["opts"])
    return state


class _DeviceArray:
    """A device view of a result's memory; keeps the result alive."""

    def __init__(self, result, ptr, count, typestr):
        self.result = result
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": typestr,
                                         "data": (ptr, False), "version": 2}


def _device_lists(state, r):
    """The answer's offsets, as the engine holds them, and its ids gathered
    into the program's table. The result lives until the next pass is done."""
    off, ids = r.device_csr()
    total = min(r.info()["total_skyline_ids"], state["ids"].numel())
    if total:
        state["ids"][:total].copy_(torch.as_tensor(_DeviceArray(r, ids, total, "<i4"), device="cuda"))
    state["result"] = r
    return {"offsets": torch.as_tensor(_DeviceArray(r, off, (1 << state["d"]) + 1, "<i8"), device="cuda"),
            "ids": state["ids"]}


def _host_lists(table, r, cuboids):
    """The ids of each cuboid, one after the other, in the program's table;
    how many each has."""
    counts, at = np.zeros(len(cuboids), np.int64), 0
    for i, c in enumerate(cuboids):
        ids = r.cuboid(c)[: table.size - at]
        table[at:at + ids.size] = ids.view(np.int32)
        counts[i] = ids.size
        at += ids.size
    return counts


def run(state):
    use = state["use"]
    if use == "serve":
        srv, reqs = state["server"], state["requests"]
        tickets = [srv.submit(q["x"], max_d=q["max_d"], subspace=q["subspace"]) for q in reqs]
        answers = []
        for t, q in zip(tickets, reqs):
            r, _ = srv.wait(t)
            answers.append({"counts": _host_lists(q["ids"], r, q["cuboids"]), "ids": q["ids"]})
            r.close()
        return answers
    if use == "host":
        ds = sk.Dataset(state["ctx"], state["x"])
        r = sk.skycube(state["ctx"], ds)
        r.download()
        counts = _host_lists(state["ids"], r, state["cuboids"])
        r.close()
        ds.close()
        return {"counts": counts, "ids": state["ids"]}
    if use == "plan":
        return _device_lists(state, state["plan"].execute())
    r = sk.skycube(state["ctx"], state["ds"], **state["opts"])
    if use == "bitmaps":
        bits, points = r.bitmaps()
        r.close()
        state["bits"][: len(bits)] = bits
        state["points"][: len(points)] = points
        return {"bits": state["bits"].view(np.int32), "points": state["points"].view(np.int32)}
    return _device_lists(state, r)


def _ids(answer):
    return int(answer["counts"].sum() if "counts" in answer else answer["offsets"][-1])


def work(case):
    """The points read once; the ids and the offsets, or the bitmaps, written
    once. How many there are follows from the data, so one pass counts them."""
    answer = run(prepare(case, 1))
    if case["use"] == "serve":
        points = sum(4 * q["n"] * q["d"] for q in _requests(case))
        out = sum(4 * _ids(a) for a in answer)
    else:
        points = 4 * case["n"] * case["d"]
        if case["use"] == "bitmaps":
            rows = int(answer["bits"].any(axis=1).sum())
            out = rows * (4 + answer["bits"].shape[1] * 4)
        else:
            out = 4 * _ids(answer) + 8 * (1 << case["d"])
    return {"bytes": points + out, "flops": 0}
