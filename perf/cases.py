"""The calls a program makes of this framework, with the sizes it makes them at.

Every case goes through the public Python API (`Engine`, `serve.Server`, `serve.serve_plain`) or
the C-ABI's device entry point (`hgx_hash_states_noalloc`), whole: inputs in, the complete result
out. A program keeps one engine and hands it one evolution (or batch, or request stream) after
another, so all inputs of one case share an engine; inputs of different seeds differ in their
vertex labels and edge order (named evolutions) or altogether (random ones). Everything computed
is whole numbers and is compared exactly.

Kinds:
  evolve    one evolution per call, the result read back to host arrays
  counts    one evolution per call, the result left on the device and its sizes returned
  requests  a list of random requests, evolved one per call
  batch     a batch of random evolutions in one call
  serve     a list of random requests through the continuous-batching server
  hash      a batch of device-resident states hashed and classified without allocation
"""
from __future__ import annotations

import ctypes
import json
import random

import numpy as np
import torch

from hypergraphrewritingengine_b200 import Engine, api, load_library, serve
from hypergraphrewritingengine_b200 import workloads as W

# --- the named rules ---------------------------------------------------------------------------

# {{x,y},{y,z}} -> {{x,y},{y,z},{z,x}} on a triangle
TRIANGLE = ([([[0, 1], [1, 2]], [[0, 1], [1, 2], [2, 0]])], [[[1, 2], [2, 3], [3, 1]]])
# {{x,y},{x,z}} -> {{x,z},{x,w},{y,w},{z,w}} on two self-loops
WPP = ([([[0, 1], [0, 2]], [[0, 2], [0, 3], [1, 3], [2, 3]])], [[[1, 1], [1, 1]]])
# {{x,y,z},{z,u,v}} -> {{w,w,y},{w,x,u},{v,u,z},{y,v,w}} on two ternary self-loops
TERNARY = ([([[0, 1, 2], [2, 3, 4]], [[5, 5, 1], [5, 0, 3], [4, 3, 2], [1, 4, 5]])],
           [[[1, 1, 1], [1, 1, 1]]])
# two rules at once (one edge grown, two edges joined) on two initial states
TWO_RULES = ([([[0, 1]], [[0, 2], [1, 2]]), ([[0, 1], [1, 2]], [[0, 2]])],
             [[[1, 2], [2, 3]], [[1, 2], [2, 3], [3, 1]]])
RULES = {"triangle": TRIANGLE, "wpp": WPP, "ternary": TERNARY, "two-rules": TWO_RULES}

# Events and states of each named evolution after 1, 2, ... steps (uncapped), for work().
GROWTH = {
    ("triangle", True): ((3, 2), (10, 4), (23, 8), (66, 13), (136, 20), (262, 30), (490, 42), (820, 57), (1315, 76)),
    ("triangle", False): ((3, 4), (18, 19), (135, 136), (1464, 1465), (22203, 22204)),
    ("wpp", True): ((2, 2), (14, 5), (68, 23), (496, 179), (5056, 1952), (66376, 26652), (1056070, 423791),
                    (18_000_000, 7_200_000)),
    ("wpp", False): ((2, 3), (26, 27), (434, 435), (9938, 9939)),
    ("ternary", True): ((2, 2), (9, 9), (86, 78), (1150, 911), (17754, 12655), (305780, 197389)),
    ("ternary", False): ((2, 3), (16, 17), (170, 171), (2544, 2545), (50004, 50005)),
    ("two-rules", True): ((9, 9), (27, 18), (82, 37), (216, 64), (458, 117), (1016, 214)),
    ("two-rules", False): ((9, 11), (47, 49), (219, 221), (1263, 1265), (8923, 8925)),
}
# Left-hand edges, arity, edges of the initial state, edges added per step, branchial pairs per event.
SHAPE = {"triangle": (2, 2, 3, 1, 3.5), "wpp": (2, 2, 2, 2, 6.3), "ternary": (2, 3, 2, 2, 3.9),
         "two-rules": (2, 2, 3, 1, 0.6)}


def listed():
    return [
        # the smallest call: an interactive step or a test, a few dozen events
        _evolve("triangle-2", "triangle", 2, quotient=False),
        # the benchmark's small configuration: every raw state kept, 22 thousand events
        _evolve("triangle-5", "triangle", 5, quotient=False),
        # several rules and roots, causal graph reduced transitively and events canonicalised (the
        # reference's defaults for its GPU entry point)
        _evolve("two-rules-reduced", "two-rules", 5, quotient=False, reduce=True, keys=3),
        # ternary hyperedges, 306 thousand events over 197 thousand classes
        _evolve("ternary-6", "ternary", 6),
        # the headline evolution, its whole result (0.9 GB) read back
        _evolve("wpp-8", "wpp", 8, cap=2_000_000, ids=False),
        # a step short of it: the ordinary large call, every array wanted
        _evolve("wpp-7", "wpp", 7),
        # the headline rule from a random start, the result left on the device
        {"name": "wpp-counts", "kind": "counts", "rule": "wpp", "edges0": 5, "steps": 7,
         "cap": 2_000_000},
        # requests as they come to a program that evolves one per call
        {"name": "requests-32", "kind": "requests", "n": 32, "cap": 4096, "set": 1},
        # the benchmark's batch: 1024 uneven evolutions in one call
        {"name": "batch-1024", "kind": "batch", "n": 1024, "cap": 4096, "edges_lo": 4,
         "edges_hi": 64, "steps_lo": 3, "steps_hi": 7, "set": 2},
        # a batch whose states are larger than a warp's lanes
        {"name": "batch-large", "kind": "batch", "n": 129, "cap": 4096, "edges_lo": 65,
         "edges_hi": 256, "steps_lo": 2, "steps_hi": 4, "set": 3},
        # continuous batching: a burst of requests admitted 50 at a time
        {"name": "serve-400", "kind": "serve", "n": 400, "cap": 4096, "per_step": 50, "set": 4},
        # states that are on the device already: hashes and classes
        {"name": "hash-200k", "kind": "hash", "n": 200_003, "arity": 2, "edges_lo": 4,
         "edges_hi": 40},
    ]


def _evolve(name, rule, steps, quotient=True, cap=0, ids=True, causal=True, branchial=True,
            reduce=False, keys=0, forwarding=0):
    c = {"kind": "evolve", "rule": rule, "steps": steps, "quotient": quotient, "cap": cap,
         "ids": ids, "causal": causal, "branchial": branchial, "reduce": reduce, "keys": keys,
         "forwarding": forwarding}
    return dict(c, name=name) if name else c


def _log(rng, lo, hi):
    """A whole number spread evenly over the logarithm of [lo, hi]."""
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


# Steps a drawn named evolution takes: quotient, full multiway.
STEPS = {"triangle": ((3, 9), (1, 5)), "wpp": ((3, 8), (2, 4)), "ternary": ((2, 6), (2, 5)),
         "two-rules": ((2, 6), (2, 5))}


def draw(rng):
    kind = rng.choice(("evolve", "evolve", "evolve", "counts", "requests", "batch", "batch",
                       "serve", "hash"))
    if kind == "evolve":
        rule = rng.choice(sorted(RULES))
        quotient = rng.random() < 0.6
        lo, hi = STEPS[rule][0 if quotient else 1]
        cap = 0 if not quotient and rng.random() < 0.5 else _log(rng, 300, 2_000_000)
        return _evolve("", rule, rng.randint(lo, hi), quotient=quotient, cap=cap,
                       ids=rng.random() < 0.5, causal=rng.random() < 0.8,
                       branchial=rng.random() < 0.8, reduce=rng.random() < 0.3,
                       keys=rng.choice((0, 0, 3, 15)), forwarding=rng.choice((0, 0, 0, 1, 2)))
    if kind == "counts":
        rule = rng.choice(("wpp", "wpp", "triangle"))
        return {"kind": kind, "rule": rule, "edges0": rng.randint(3, 8 if rule == "wpp" else 6),
                "steps": rng.randint(3, 7),
                "cap": _log(rng, 1000, 2_000_000 if rule == "wpp" else 100_000)}
    one = rng.randrange(1, 1 << 30)   # which random evolutions
    if kind == "requests":
        return {"kind": kind, "n": _log(rng, 2, 40), "cap": _log(rng, 256, 16384), "set": one}
    if kind == "batch":
        n = _log(rng, 8, 1024)
        cap = _log(rng, 256, min(65536, 4096 * 1024 // n))
        if rng.random() < 0.3:
            return {"kind": kind, "n": min(n, 200), "cap": min(cap, 4096), "edges_lo": 65,
                    "edges_hi": rng.randint(100, 256), "steps_lo": 2, "steps_hi": rng.randint(3, 4),
                    "set": one}
        return {"kind": kind, "n": n, "cap": cap, "edges_lo": 4, "edges_hi": rng.randint(12, 64),
                "steps_lo": rng.randint(2, 3), "steps_hi": rng.randint(5, 7), "set": one}
    if kind == "serve":
        return {"kind": kind, "n": _log(rng, 16, 400), "cap": _log(rng, 512, 4096),
                "per_step": _log(rng, 4, 400), "set": one}
    return {"kind": "hash", "n": _log(rng, 64, 524_288), "arity": rng.choice((2, 3)),
            "edges_lo": rng.randint(1, 8), "edges_hi": rng.randint(12, 64)}


# --- inputs ------------------------------------------------------------------------------------

_kept = {}   # the engine a program keeps for its calls of one kind


def _engine(case):
    key = json.dumps({k: v for k, v in case.items() if k != "name"}, sort_keys=True)
    if key not in _kept:
        for old in _kept.values():
            old.close()
        _kept.clear()
        eng = Engine(0, causal=case.get("causal", True), branchial=case.get("branchial", True))
        eng.set_option(api.OPT_KEEP_STATE_EDGE_IDS, case.get("ids", True))
        eng.set_option(api.OPT_TRANSITIVE_REDUCTION, case.get("reduce", False))
        eng.set_option(api.OPT_EVENT_SIGNATURE_KEYS, case.get("keys", 0))
        eng.set_option(api.OPT_FORWARDING, case.get("forwarding", 0))
        _kept[key] = eng
    return _kept[key]


def _relabelled(roots, rng, shuffle=False):
    """The same initial states under other vertex labels (and their edges in another order)."""
    vertices = sorted({v for st in roots for e in st for v in e})
    label = dict(zip(vertices, rng.sample(range(1, 100_000), len(vertices))))
    out = []
    for st in roots:
        st = [[label[v] for v in e] for e in st]
        if shuffle:
            rng.shuffle(st)
        out.append(st)
    return out


def _evolutions(case, seed):
    """The case's random evolutions, relabelled and in an order of the seed's own."""
    at = W.SplitMix64(case["set"]).next() >> 1
    if case["kind"] == "batch":
        evs = [W.random_evolution(i, seed=at, max_states=case["cap"], edges_lo=case["edges_lo"],
                                  edges_hi=case["edges_hi"], steps_lo=case["steps_lo"],
                                  steps_hi=case["steps_hi"]) for i in range(case["n"])]
    else:
        # the served workload's requests: initial edges lognormal (median 16, at most 256), 2-8 steps
        evs = [W.random_evolution(i, seed=at, max_states=case["cap"], edges_lo=4, steps_lo=2,
                                  steps_hi=8, lognormal_median=16.0, lognormal_max=256)
               for i in range(case["n"])]
    rng = random.Random(seed)
    for ev in evs:
        ev.roots = _relabelled(ev.roots, rng)
    rng.shuffle(evs)
    return evs


def _hash_inputs(case, seed):
    """Device-resident state records (edge ids | arities packed four per word | vertices): connected
    random states, half of them relabelled copies of others, as the children of an evolution are."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    n, a, lo, hi = case["n"], case["arity"], case["edges_lo"], case["edges_hi"]
    base = (n + 1) // 2

    def below(m, *shape):
        return (torch.rand(shape, generator=g, device="cuda", dtype=torch.float64) * m).long()

    ne_b = lo + below(hi - lo + 1, base)
    nv_b = torch.clamp((ne_b + 1) // 2, min=3)
    # edge j of the chain joins vertices j and j + 1; the others are uniform
    v = below(nv_b[:, None, None], base, hi, a)
    chain = torch.arange(hi, device="cuda")[None, :] < nv_b[:, None] - 1
    j = torch.arange(hi, device="cuda")[None, :].expand(base, hi)
    v[:, :, 0] = torch.where(chain, j, v[:, :, 0])
    v[:, :, 1] = torch.where(chain, j + 1, v[:, :, 1])
    src = torch.cat([torch.arange(base, device="cuda"), below(base, n - base)])
    ne = ne_b[src]
    # labels: an odd multiplier and an offset per state, so copies carry other labels
    v = (v[src] * (2 * below(1 << 12, n) + 1)[:, None, None] + below(1 << 16, n)[:, None, None]) % (1 << 20)
    aw = (ne + 3) // 4
    words = ne + aw + ne * a
    off = torch.cumsum(words, 0) - words
    rec = torch.zeros(int(words.sum()), dtype=torch.int32, device="cuda")
    k = torch.arange(hi, device="cuda")[None, :]
    live = k < ne[:, None]
    first = torch.cumsum(ne, 0) - ne
    rec[(off[:, None] + k)[live]] = (first[:, None] + k)[live].int()
    rec.index_put_(((off[:, None] + ne[:, None] + k // 4)[live],),
                   (a << (8 * (k % 4))).expand(n, hi)[live].int(), accumulate=True)
    p = torch.arange(a, device="cuda")
    at = (off + ne + aw)[:, None, None] + k[:, :, None] * a + p
    rec[at[live]] = v[live].int()
    return {"rec": rec, "off": off.long(), "ne": ne.int(), "nocc": (ne * a).int(), "n": n,
            "max_ne": hi, "max_nocc": hi * a,
            "hash": torch.empty(n, dtype=torch.int64, device="cuda"),
            "cls": torch.empty(n, dtype=torch.int32, device="cuda")}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "hash":
        return dict(_hash_inputs(case, seed), kind=kind, lib=load_library())
    s = {"kind": kind, "eng": _engine(case)}
    if kind in ("evolve", "counts"):
        rules, roots = RULES[case["rule"]]
        if kind == "counts":
            start = W.SplitMix64(W.SplitMix64(seed).next())
            roots = [W.random_hypergraph(start, case["edges0"], 2)]
        quotient = case.get("quotient", True)
        s.update(rules=rules, roots=_relabelled(roots, random.Random(seed), not quotient and not case["cap"]),
                 steps=case["steps"], quotient=quotient, cap=case["cap"])
        return s
    evs = _evolutions(case, seed)
    if kind == "batch":
        s["evolutions"] = evs
        s["jobs"], s["blobs"] = Engine.make_jobs(evs)
    else:
        s["arrivals"] = [(0.0, ev) for ev in evs]
        s["per_step"] = case.get("per_step", 0)
    return s


# --- one pass ----------------------------------------------------------------------------------

ARRAYS = ("state_hash", "state_depth", "events", "causal", "branchial", "event_cons_off",
          "event_cons", "event_prod", "state_edge_off", "state_edge_ids", "state_arity",
          "state_vert_off", "state_verts", "event_signature")


def _signed(a):
    """The same bytes as signed words (64-bit hashes, 32-bit ids)."""
    return a if a.dtype.itemsize == 1 else a.view(np.int64 if a.dtype.itemsize == 8 else np.int32)


class Results(dict):
    """The results of many evolutions, by array name: reading a name joins that array over all of
    them in input order. The results themselves are what the pass returned."""

    def __init__(self, results):
        super().__init__((name, None) for name in ARRAYS + ("sizes",))
        self.results = results

    def __getitem__(self, name):
        if name == "sizes":
            return np.array([[r.num_classes, r.num_canonical_events, int(r.truncated)] +
                             [len(getattr(r, x)) for x in ARRAYS] for r in self.results], np.int64)
        return np.concatenate([_signed(getattr(r, name)) for r in self.results])


def run(state):
    kind = state["kind"]
    if kind == "hash":
        p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
        status = state["lib"].hgx_hash_states_noalloc(
            p(state["rec"]), p(state["off"]), p(state["ne"]), p(state["nocc"]), state["n"],
            state["max_ne"], state["max_nocc"], p(state["hash"]), p(state["cls"]),
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if status:
            raise RuntimeError(state["lib"].hgx_last_error().decode())
        return {"hash": state["hash"], "class": state["cls"]}
    eng = state["eng"]
    if kind == "evolve":
        return Results([eng.evolve(state["rules"], state["roots"], state["steps"],
                                   quotient=state["quotient"], max_states=state["cap"])])
    if kind == "counts":
        return {k: int(v) for k, v in eng.counts(state["rules"], state["roots"], state["steps"],
                                                 quotient=True, max_states=state["cap"]).items()}
    if kind == "batch":
        return Results(eng.evolve_batch(state["evolutions"], state["jobs"]))
    if kind == "requests":
        recs = serve.serve_plain(eng, state["arrivals"], realtime=False)
    else:
        recs = serve.Server(eng).run(state["arrivals"], realtime=False,
                                     admit_per_step=state["per_step"])
    return Results([r.result for r in recs])


# --- what a pass cannot do without ---------------------------------------------------------------

def work(case):
    """Bytes of the inputs and of the result records, each once (integer work: no flops)."""
    kind = case["kind"]
    if kind == "hash":
        edges = (case["edges_lo"] + case["edges_hi"]) / 2
        # a record's edge ids, arities and vertices, its offset and sizes; a hash and a class
        return {"bytes": case["n"] * (edges * (5 + 4 * case["arity"]) + 16 + 12), "flops": 0}
    if kind in ("evolve", "counts"):
        lhs, arity, e0, grow, pairs = SHAPE[case["rule"]]
        e0 = case.get("edges0", e0)
        steps, cap = case["steps"], case["cap"]
        if kind == "counts":   # a random start grows like a named one that is a step or two ahead
            rows = GROWTH[(case["rule"], True)]
            events, states = rows[min(steps + 1, len(rows)) - 1]
            if case["rule"] == "triangle":
                events, states = 10 ** (steps - 2), 6 ** (steps - 2)
        else:
            events, states = GROWTH[(case["rule"], case["quotient"])][steps - 1]
        if cap and states > cap:
            events, states = events * cap / states, cap
        edges = e0 + grow * steps
        b = events * (16 + 4 + 8 + 4 * lhs) + states * 12
        b += events * 24 if case.get("causal", True) else 0
        b += events * pairs * 8 if case.get("branchial", True) else 0
        b += states * (8 + edges * (1 + 4 * arity + (4 if case.get("ids", True) else 0)))
        b += 8 * events if case.get("keys", 0) else 0
        return {"bytes": max(b, 256), "flops": 0}
    # random evolutions: the mean result of one (measured), growing with its cap and its states
    if kind == "batch":
        one = 1.6e6 if case["edges_hi"] > 64 else 6.6e5 * case["edges_hi"] / 64
    else:
        one = 4.4e5
    return {"bytes": case["n"] * one * (case["cap"] / 4096) ** 0.5, "flops": 0}


def tolerance(case):
    return "exact"   # whole numbers throughout: ids, counts and 64-bit hashes
