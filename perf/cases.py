"""Timed cases of the sbfs engine: what its users have it do, through its public entry points.

A case is a dict of plain values.  ``kind`` says which call a pass makes:

  device   ``Engine.solve_device`` + ``wait_device`` on records in HBM
  host     ``Engine.solve`` on host buffers (lengths and words)
  verify   ``Engine.verify`` on host buffers (lengths and the first violation)
  serving  ``Server.submit_many`` of a burst, then ``poll_array`` until every result is back

and ``batch`` what it is given:

  uniform  ``count`` automata of ``n`` states with uniform random maps, from the
           .NET ``System.Random`` batch generator, in tight 2n-byte records
  mixed    ``count`` automata, sizes uniform (``log`` = False) or log-uniform in
           ``lo..hi``, one in ``cerny_every`` a Cerny automaton, 64-byte records
  large    for each size in ``sizes``: ``count`` random automata, the Cerny
           automaton and a random permutation plus one merge, 64-byte records

Every output is a whole number (lengths, word bits, an index), so there is no
``exact``.  Where several words are equally short and the kernels race for
which one is found (n > 14), the cases ask for lengths, as the reference's
``Verify`` does; the serving results always carry their words.
"""
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(1, os.path.join(ROOT, "gpgpu-binary-automaton-synchronizing-algorithms_b200"))

import sbfs  # noqa: E402
from sbfs import dotnet_random  # noqa: E402
from sbfs import problem as P  # noqa: E402
from sbfs.server import Server  # noqa: E402


def listed():
    return [
        # one automaton through the host call: all latency (an interactive check, a C# caller's single Problem)
        dict(name="n12 one host", kind="host", batch="uniform", n=12, count=1, pinned=False, words=True),
        # the plain configuration: 10,000 automata of 8 states in numpy buffers
        dict(name="n8 10k host", kind="host", batch="uniform", n=8, count=10_000, pinned=False, words=True),
        # an odd batch with a record stride that is no multiple of four, resident on the GPU
        dict(name="n10 77777 device", kind="device", batch="uniform", n=10, count=77_777, words=True, graph=False),
        # the headline batch, device-resident
        dict(name="n12 1M device", kind="device", batch="uniform", n=12, count=1_000_000, words=True, graph=False),
        # the headline batch end to end from pinned host buffers
        dict(name="n12 1M host", kind="host", batch="uniform", n=12, count=1_000_000, pinned=True, words=True),
        # the reference's published configuration: one Verify call over 2^21 automata of 13 states, numpy buffers
        dict(name="n13 2M verify", kind="verify", batch="uniform", n=13, count=1 << 21, pinned=False, words=False),
        # the sizes above the benchmark's, up to the largest that stays on chip
        dict(name="n14 500k device", kind="device", batch="uniform", n=14, count=500_000, words=True, graph=False),
        dict(name="n16 200k device", kind="device", batch="uniform", n=16, count=200_000, words=False, graph=False),
        dict(name="n20 30k device", kind="device", batch="uniform", n=20, count=30_000, words=False, graph=False),
        # the mixed configuration: sizes 6..20, 1 % Cerny automata, replayed from a CUDA graph
        dict(name="mixed 200k device", kind="device", batch="mixed", lo=6, hi=20, log=False, count=200_000,
             cerny_every=100, words=False, graph=True),
        # the large configuration: n = 24, 26, 28 with 2^n-bit visited sets, one Verify call
        dict(name="large 24 26 28", kind="verify", batch="large", sizes="24,26,28", count=64, pinned=False,
             words=False),
        # a burst of single-automaton requests to the serving loop, n log-uniform in 8..24, 5 % Cerny
        dict(name="serving 10k burst", kind="serving", batch="mixed", lo=8, hi=24, log=True, count=10_000,
             cerny_every=20),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["uniform"] * 5 + ["mixed", "mixed", "large", "serving"])
    if kind == "uniform":
        n = rng.randint(4, 20)
        most = 1 << 20 if n <= 14 else 1 << 17 if n <= 16 else 1 << 15
        call = rng.choice(["device", "host", "verify"])
        c = dict(kind=call, batch="uniform", n=n, count=_log_int(rng, 1, most))
        c["words"] = call == "host" and n <= 14 or call == "device" and n <= 14 and rng.random() < 0.5
        if call == "host" and not c["words"]:
            c["kind"] = "verify"
        if c["kind"] == "device":
            c["graph"] = rng.random() < 0.5
        else:
            c["pinned"] = rng.random() < 0.5
        return c
    if kind == "mixed":
        lo, hi = sorted(rng.sample(range(4, 21), 2))
        return dict(kind="device", batch="mixed", lo=lo, hi=hi, log=False, count=_log_int(rng, 500, 200_000),
                    cerny_every=rng.choice([50, 100, 400]), words=False, graph=rng.random() < 0.5)
    if kind == "large":
        sizes = sorted(rng.sample(range(21, 28), rng.randint(1, 2)))
        return dict(kind="verify", batch="large", sizes=",".join(map(str, sizes)), count=_log_int(rng, 4, 64),
                    pinned=rng.random() < 0.5, words=False)
    return dict(kind="serving", batch="mixed", lo=rng.randint(4, 8), hi=rng.randint(16, 23), log=True,
                count=_log_int(rng, 100, 10_000), cerny_every=20)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _mixed_batch(case, seed):
    """(records, sizes) on the GPU: random maps of random sizes, every
    cerny_every-th automaton a Cerny one."""
    dev, count = torch.device("cuda"), case["count"]
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    u = torch.rand(count, device=dev, generator=g, dtype=torch.float64)
    lo, hi = case["lo"], case["hi"]
    if case["log"]:
        ns = torch.floor(lo * ((hi + 1) / lo) ** u)
    else:
        ns = torch.floor(lo + u * (hi + 1 - lo))
    ns = ns.clamp(lo, hi).to(torch.int64)
    state = torch.arange(32, device=dev)
    maps = torch.floor(torch.rand((count, 2, 32), device=dev, generator=g) * ns[:, None, None]).to(torch.int64)
    maps = torch.minimum(maps, ns[:, None, None] - 1)
    # C_n: a is the cycle, b sends 0 to 1 and fixes the rest
    at = torch.arange(int(seed) % case["cerny_every"], count, case["cerny_every"], device=dev)
    maps[at, 0] = (state + 1) % ns[at, None]
    maps[at, 1] = torch.where(state == 0, 1, state)
    maps = torch.where(state < ns[:, None, None], maps, 0)
    return maps.reshape(count, 64).to(torch.uint8).contiguous(), ns.to(torch.uint8)


def _large_batch(case, seed):
    rows, ns = [], []
    for n in map(int, case["sizes"].split(",")):
        rows += [P.uniform_maps(case["count"], n, seed + n), P.cerny_record(n)[None], P.perm_merge_record(n, seed + 99 + n)[None]]
        ns += [n] * (case["count"] + 2)
    return np.concatenate(rows), np.array(ns, dtype=np.uint8)


def _batch(case, seed):
    """(records, sizes or None, n, lstride, largest n) with the records in host memory."""
    if case["batch"] == "uniform":
        n = case["n"]
        recs = dotnet_random.fill_array_of_problems(case["count"], n, seed & 0x7FFFFFFF, lstride=n)
        return recs, None, n, n, n
    recs, ns = _large_batch(case, seed) if case["batch"] == "large" else [t.cpu().numpy() for t in _mixed_batch(case, seed)]
    return recs, ns, 0, 32, int(ns.max())


def _automata(case):
    return (case["count"] + 2) * len(case["sizes"].split(",")) if case["batch"] == "large" else case["count"]


# a program keeps one engine (and one server) for all its batches
_engines, _servers = {}, {}


def _engine(graph=False):
    if graph not in _engines:
        _engines[graph] = sbfs.Engine(device=0, use_graph=graph)
    return _engines[graph]


def _server():
    if 0 not in _servers:
        _servers[0] = Server(device=0)
    return _servers[0]


def _pin(a):
    return torch.from_numpy(a).pin_memory().numpy()


def prepare(case, seed):
    recs, ns, n, lstride, max_n = _batch(case, seed)
    s = dict(kind=case["kind"], n=n, lstride=lstride, max_n=max_n, count=recs.shape[0])
    if case["kind"] == "serving":
        s.update(server=_server(), recs=recs, ns=ns)
        return s
    s["ws"] = ws = sbfs.word_stride_for(max_n)
    if case["kind"] == "device":
        dev = torch.device("cuda")
        s.update(engine=_engine(case["graph"]), recs=torch.from_numpy(recs).to(dev),
                 ns=None if ns is None else torch.from_numpy(ns).to(dev),
                 len=torch.empty(s["count"], dtype=torch.int32, device=dev),
                 words=torch.empty((s["count"], ws), dtype=torch.int64, device=dev) if case["words"] else None,
                 fv=torch.empty(1, dtype=torch.int64, device=dev))
        return s
    out_len = np.empty(s["count"], dtype=np.int32)
    out_words = np.empty((s["count"], ws), dtype=np.uint64)
    if case["pinned"]:
        recs, out_len = _pin(recs), _pin(out_len)
        out_words = _pin(out_words.view(np.int64)).view(np.uint64)
    s.update(engine=_engine(), recs=recs, ns=ns, out=(out_len, out_words))
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def _run_serving(s):
    srv, count = s["server"], s["count"]
    ids = srv.submit_many(s["recs"], s["ns"])
    parts, left = [], count
    while left:
        part = srv.poll_array(timeout_ms=1000)
        parts.append(part)
        left -= len(part)
    res = np.concatenate(parts)
    res = res[np.argsort(res["id"])]
    return {"order": (res["id"] - ids).astype(np.int64), "status": res["status"], "len": res["len"], "n": res["n"],
            "word": res["word"].astype(np.int64)}


def run(s):
    if s["kind"] == "serving":
        return _run_serving(s)
    eng = s["engine"]
    if s["kind"] == "device":
        eng.solve_device(s["recs"], s["lstride"], s["count"], n=s["n"], d_ns=s["ns"], max_n=s["max_n"],
                         d_len=s["len"], d_words=s["words"], word_stride=s["ws"] if s["words"] is not None else 0,
                         d_first_violation=s["fv"])
        eng.wait_device()
        return [s["len"], s["words"], s["fv"]]
    if s["kind"] == "host":
        r = eng.solve(s["recs"], ns=s["ns"], n=s["n"], lstride=s["lstride"], out=s["out"])
        return [r["len"], r["words"].view(np.int64), r["first_violation"]]
    r = eng.verify(s["recs"], ns=s["ns"], n=s["n"], lstride=s["lstride"])
    return [r["len"], r["first_violation"]]


def work(case):
    """Every record read once, every length (and word) written once."""
    count = _automata(case)
    if case["batch"] == "uniform":
        rec, max_n = 2 * case["n"], case["n"]
    else:
        rec, max_n = 65, int(case["sizes"].split(",")[-1]) if case["batch"] == "large" else case["hi"]
    out = 4 + (8 * sbfs.word_stride_for(max_n) if case.get("words") or case["kind"] == "serving" else 0)
    return {"bytes": count * (rec + out) + 8, "flops": 0}
