"""What a program that uses this engine has it do, as cases whose passes can be timed.

Every case goes through the public binding (``six-one-five_b200/s615.py`` over
the C ABI of ``include/s615.h``): host units in, raw hits, counters and verified
identities out, or a table built.  The kinds:

  units   s615_run of Stage-1 units of classes 2-5 against a resident table,
          then s615_verify of the hits: what one chunk of a campaign is.
          ``share`` is the mix: 5 for class 5 alone, 0 for the mixed stream.
  band    s615_prepare_band + run of every class-5 unit of a B range (the
          units are made on the device).
  jobs    the reduced-T jobs of a .bbj file (kind 2 units), run and verified.
  c617    (6,1,7) class-5 candidates of one B;  j617: its class 1-4 jobs.
  build   a pair table built and asked for keys;  export: also read back to
          the host, as the table builder does before it writes the file.
  serve   requests through the serving loop: start, submit, poll, stop.

Sizes follow bench.py (config 1, the 3.2M class-5 band, the mixed stream, the
job stream, the (6,1,7) band at 400k, 50-unit serving requests) and the tables
that they need (N = ceil(B / 42)); fewer units where a whole band takes longer
than a second or two.  A program loads its table once and keeps it, so the
process keeps the table of the last case.
"""
import math
import os
import random
import sys

import numpy as np

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "six-one-five_b200"))
import s615  # noqa: E402
import workloads as W  # noqa: E402


def listed():
    return [
        # Config 1: every class-5 unit of B in [1000, 30000] with 8 plants, a table that fits the
        # cache many times over.  The smallest call: launches and host work.
        {"name": "config1", "kind": "units", "share": 5, "B_lo": 1000, "B_hi": 30000, "n": 0,
         "plants": 8, "N": 715, "r": 48, "layout": 0, "shards": 1, "flags": 0},
        # One 50-unit request of the 3.2M band: the latency of a call that cannot fill the GPU long.
        {"name": "request50", "kind": "units", "share": 5, "B_lo": 3200000, "B_hi": 3220000,
         "n": 50, "plants": 1, "N": 76667, "r": 48, "layout": 0, "shards": 1, "flags": 0},
        # A chunk of the 3.2M class-5 band, the headline workload: the largest table and call.
        {"name": "band_3200k", "kind": "units", "share": 5, "B_lo": 3200000, "B_hi": 3220000,
         "n": 12000, "plants": 8, "N": 76667, "r": 48, "layout": 0, "shards": 1, "flags": 0},
        # A class-5 band at 1M, units made on the device (Stage-1 on the GPU), N = 24,000.
        {"name": "band_1000k", "kind": "band", "B_lo": 1000000, "B_hi": 1007999, "width": 2400,
         "N": 24000, "r": 48, "layout": 0, "shards": 1, "flags": 0},
        # The sharper gate (opt-in) on a class-5 chunk: sieve bound, few probes.
        {"name": "sharp_2000k", "kind": "units", "share": 5, "B_lo": 1900000, "B_hi": 2000000,
         "n": 6001, "plants": 8, "N": 48000, "r": 48, "layout": 0, "shards": 1, "flags": 8},
        # The mixed-class stream (2:4%, 3:1%, 4:48%, 5:47%), heavy-tailed extents.
        {"name": "mixed_2000k", "kind": "units", "share": 0, "B_lo": 1000000, "B_hi": 2000000,
         "n": 6000, "plants": 16, "N": 48000, "r": 48, "layout": 0, "shards": 1, "flags": 0},
        # Reduced-T jobs of classes 1-4 (a .bbj file's content): many small units.
        {"name": "jobs_2000k", "kind": "jobs", "B_lo": 1000000, "B_hi": 2000000, "n": 1501,
         "N": 48000, "r": 48, "layout": 0, "shards": 1, "flags": 0},
        # Serving: 24 requests of 50 mixed units, B uniform on [1M, 2M].
        {"name": "serve_2000k", "kind": "serve", "B_lo": 1000000, "B_hi": 2000000, "n": 24,
         "N": 48000, "r": 48, "layout": 0, "shards": 1, "flags": 0},
        # (6,1,7) class 5 at the 400k band, a part of one B's candidates.
        {"name": "c617_400k", "kind": "c617", "B_lo": 400000, "B_hi": 440000, "n": 100,
         "N": 10476, "r": 48, "layout": 0, "shards": 1, "flags": 0},
        # (6,1,7) classes 1-4 at the same band: a part of one B's find4 jobs.
        {"name": "j617_400k", "kind": "j617", "B_lo": 400000, "B_hi": 440000, "n": 100001,
         "N": 10476, "r": 48, "layout": 0, "shards": 1, "flags": 0},
        # Table builds: the search table of B <= 2M, and a small one read back whole.
        {"name": "build_48k", "kind": "build", "N": 48000, "r": 48, "layout": 0},
        {"name": "export_6k", "kind": "export", "N": 6000, "r": 48, "layout": 0},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _points5(B):
    """R > 0 grid points of one class-5 unit: 6 x 4 residues of the (B/14) x (B/21) grid."""
    return 24 / 46656 * B * B / 294 * 0.91 + 1


def _jobs234(B):
    """Free-term values of an average class 2-4 unit of the mixed stream."""
    return (4 * B / 1701 + 1 * B / 336 + 48 * B / 13600) / 53 + 1


def draw(rng):
    kind = rng.choice(["units"] * 4 + ["mixed"] * 3 + ["band", "band", "jobs", "serve", "c617",
                                                       "j617", "build", "export"])
    r, layout, shards = rng.choice([48, 48, 48, 48, 32]), rng.choice([0, 0, 0, 0, 1]), 1
    if kind in ("build", "export"):
        return {"kind": kind, "N": _log(rng, 2000, 48000) if kind == "build" else _log(rng, 700, 6000),
                "r": r, "layout": layout}
    if kind in ("c617", "j617"):
        B = _log(rng, 40000, 430000)
        c = {"kind": kind, "B_lo": B, "B_hi": B + B // 40,
             "n": rng.randint(1, 100) if kind == "c617" else _log(rng, 100, 100000)}
    elif kind == "band":
        B = _log(rng, 60000, 3100000)
        most = min(6000, max(1, int(2.0e11 / (7.77 * _points5(B)))))   # about 7.8 units a B
        width = _log(rng, 1, most)
        c = {"kind": "band", "B_lo": B, "B_hi": B + max(width, B // 100), "width": width}
    elif kind == "jobs":
        B = _log(rng, 60000, 1800000)
        c = {"kind": "jobs", "B_lo": B, "B_hi": B + B // 10, "n": _log(rng, 10, 1500)}
    elif kind == "serve":
        B = _log(rng, 60000, 2800000)
        c = {"kind": "serve", "B_lo": B, "B_hi": B + B // 10, "n": rng.randint(1, 24)}
    else:
        B = _log(rng, 30000, 3000000)
        most = min(20000, max(8, int(1.9e11 / _points5(B))))
        c = {"kind": "units", "share": 0 if kind == "mixed" else 5, "B_lo": B, "B_hi": B + B // 16,
             "n": _log(rng, 1, most), "plants": rng.choice([0, 1, 7])}
        if rng.random() < 0.1:
            shards = rng.choice([2, 3])
    c.update({"N": -(-c["B_hi"] // 42), "r": r, "layout": layout, "shards": shards,
              "flags": rng.choice([0] * 7 + [8])})
    return c


# ---- the resident table ------------------------------------------------------
_kept = {"engine": None, "key": None, "tid": None}


def _engine():
    if _kept["engine"] is None:
        _kept["engine"] = s615.Engine(0)
    return _kept["engine"]


def _drop_table():
    if _kept["tid"] is not None:
        _engine().free_table(_kept["tid"])
        _kept["tid"] = _kept["key"] = None


def _table(case):
    key = (case["N"], case["r"], case["layout"], case["shards"])
    if _kept["key"] != key:
        _drop_table()
        eng = _engine()
        if case["shards"] > 1:
            _kept["tid"] = eng.build_table_sharded(case["N"], case["r"], case["shards"], case["layout"])
        else:
            _kept["tid"] = eng.build_table(case["N"], case["r"], case["layout"])
        _kept["key"] = key
    return _kept["tid"]


# ---- inputs --------------------------------------------------------------------
def _seed32(seed):
    return int(seed) % (2**32)


def _units5(case, seed):
    """n class-5 units of the range: a run of consecutive B from a seeded start, as a
    campaign's chunk is (n = 0: the whole range)."""
    lo, hi, n = case["B_lo"], case["B_hi"], case["n"]
    if n == 0:
        return W.cls5_units(lo, hi)
    B = random.Random(seed).randint(lo, hi)
    out = []
    while len(out) < n:
        if W.eligible(B):
            out += [(B, u) for u in s615.unit_candidates(B, 5)]
        B = B + 1 if B < hi else lo
    return out[:n]


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("build", "export"):
        _drop_table()
        rng, N = np.random.RandomState(_seed32(seed)), case["N"]
        i = rng.randint(1, N + 1, size=(2, 1 << 19)).astype(np.uint64)
        with np.errstate(over="ignore"):
            member = i[0] ** np.uint64(6) + i[1] ** np.uint64(6)
        other = rng.randint(0, 2**63, size=1 << 19, dtype=np.int64).astype(np.uint64) * np.uint64(2)
        keys = np.concatenate([member, other])
        rng.shuffle(keys)
        return {"kind": kind, "engine": _engine(), "N": N, "r": case["r"], "layout": case["layout"],
                "keys": keys}
    st = {"kind": kind, "engine": _engine(), "tid": _table(case), "N": case["N"],
          "flags": case["flags"]}
    lo, hi, sd = case["B_lo"], case["B_hi"], _seed32(seed)
    if kind == "units" and case["share"] == 5:
        st["units"], st["n"] = W.unit_array(_units5(case, seed),
                                            W.plants(case["plants"], sd, lo, hi, case["N"]), case["N"])
    elif kind == "units":
        p = case["plants"]
        st["units"], st["n"] = W.mixed_unit_array(
            W.mixed_units(case["n"], sd, lo, hi), W.plants(p // 2, sd, lo, hi, case["N"]),
            W.plants234(p - p // 2, sd, lo, hi, case["N"]), case["N"])
    elif kind == "band":
        st["B_lo"] = random.Random(seed).randint(lo, max(lo, hi - case["width"] + 1))
        st["B_hi"] = st["B_lo"] + case["width"] - 1
    elif kind == "jobs":
        units = W.mixed_units(case["n"], sd, lo, hi, mix={1: 0.01, 2: 0.08, 3: 0.01, 4: 0.90})
        st["units"], st["n"], _ = s615.expand_units(units)
    elif kind == "serve":
        st["requests"] = []
        for q in range(case["n"]):
            u = W.mixed_units(49, (sd + 7919 * q) % 2**32, lo, hi, log_uniform=False)
            st["requests"].append(W.mixed_unit_array(
                u, W.plants(1, (sd + 7919 * q) % 2**32, lo, hi, case["N"]), [], case["N"]))
    else:
        rng = random.Random(seed)
        picked, B = [], rng.randint(lo, hi)
        while True:
            B = B + 1 if B < hi else lo
            if not W.eligible(B):
                continue
            arr, n = s615.candidates617(B) if kind == "c617" else s615.jobs617_band([B], (1, 2, 3, 4))
            if n:
                at = rng.sample(range(n), min(n, case["n"])) if kind == "c617" else None
                first = rng.randint(0, n - min(n, case["n"])) if at is None else 0
                picked = at if at is not None else range(first, first + min(n, case["n"]))
                break
        out = (s615.Unit * len(picked))()
        for k, i in enumerate(picked):
            out[k] = arr[i]
        st["units"], st["n"] = out, len(picked)
    return st


# ---- one pass --------------------------------------------------------------------
def _rows(a):
    """a with zero rows up to a multiple of 64: the number of hits is not known beforehand."""
    out = np.zeros((-(-max(len(a), 1) // 64) * 64, a.shape[1]), dtype=a.dtype)
    out[:len(a)] = a
    return out


def _hits(h):
    """The raw hits (an unordered list) by fingerprint, as rows of 32-bit words."""
    return h[np.argsort(h["fp"], kind="stable")].view("<u4").reshape(-1, 8)


def _counters(c):
    return np.array([c.calls, c.gated, c.probes, c.pos, c.hits, c.tri_total, c.tri_skipped],
                    dtype=np.int64)


def _solutions(sols):
    return np.array([(s.unit, s.kind, s.cls, s.d, s.e, s.c1, s.c2, s.c3, s.c4) for s in sols],
                    dtype=np.int64).reshape(-1, 9)


def run(st):
    eng, kind = st["engine"], st["kind"]
    if kind == "build":
        tid = eng.build_table(st["N"], st["r"], st["layout"])
        h = eng.table_info(tid).hdr
        found = eng.query(tid, st["keys"])
        eng.free_table(tid)
        return {"found": found, "header": [h.n_keys, h.m_cells, h.mix_seed, h.N]}
    if kind == "export":
        tid = eng.build_table(st["N"], st["r"], st["layout"])
        header, cells = eng.export_table(tid)
        found = eng.query(tid, st["keys"])
        eng.free_table(tid)
        return {"cells": cells, "found": found, "header": np.frombuffer(header, dtype=np.uint8)}
    if kind == "serve":
        eng.serve_start(2)
        tickets = [eng.submit(st["tid"], u, n, st["flags"]) for u, n in st["requests"]]
        done = {}
        while len(done) < len(tickets):
            for x in eng.poll(64, 1000):
                done[x["ticket"]] = x
        eng.serve_stop()
        res = [done[t] for t in tickets]
        return {"hits": _rows(np.concatenate([_hits(x["hits"]) for x in res])),
                "solutions": _rows(np.concatenate([_solutions(x["solutions"]) for x in res])),
                "status": [x["status"] for x in res]}
    if kind == "band":
        units, n, hits, ctr = eng.run_band(st["tid"], st["B_lo"], st["B_hi"], st["flags"])
    else:
        units, n = st["units"], st["n"]
        hits, ctr = eng.run(st["tid"], units, n, st["flags"])
    sols = eng.verify(units, n, hits, st["N"]) if len(hits) else []
    return {"hits": _rows(_hits(hits)), "counters": _counters(ctr),
            "solutions": _rows(_solutions(sols))}


# ---- what a pass cannot do without -------------------------------------------------
def work(case):
    """bytes: the unit records (72 B) and the three r-bit cells of every point that passes the
    gate (2.7% of the points, 18% in the (6,1,7) search, 0.19% with the sharper gate), or a
    build's keys once and its cells once; flops: one gate decision a point, or the three cells of a key (integer work)."""
    kind, r = case["kind"], case["r"]
    if kind in ("build", "export"):
        n = case["N"] ** 2 / 2
        return {"bytes": n * 8 + 1.23 * n * r / 8, "flops": 3 * n}
    B = 0.5 * (case["B_lo"] + case["B_hi"])
    lim = B / 42
    row = 0.167 * 0.9 * lim   # c3 values of an average find3 row
    if kind == "units":
        n = case["n"] or 725
        points = n * (_points5(B) if case["share"] == 5
                      else 0.47 * _points5(B) + 0.53 * _jobs234(B) * row)
    elif kind == "serve":
        n = 50 * case["n"]
        points = n * (0.47 * _points5(B) + 0.53 * _jobs234(B) * row)
    elif kind == "band":
        n = case["width"] * 2 / 7 * max(1.0, B / 117649)   # eligible B, their units
        points = n * _points5(B)
    elif kind == "jobs":
        n = case["n"] * B / 10000
        points = n * row
    else:   # (6,1,7): rows d (or one job), c4 windows that pass the triple gate, c3 windows
        n = case["n"]
        rows = B / 21 / 64 * 4 if kind == "c617" else 1
        points = n * rows * 0.35 * 0.167 * lim * row * (0.19 if kind == "c617" else 0.15)
    gate = 0.0019 if case["flags"] & 8 else 0.18 if kind in ("c617", "j617") else 0.027
    cells = 3 * r / 8 * points * gate
    return {"bytes": 72 * n + cells + 8, "flops": points}
