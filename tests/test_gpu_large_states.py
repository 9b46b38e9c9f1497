"""Evolutions of states past 256 edges (positions of more than a byte) against the oracle."""
import ctypes
import time

import numpy as np
import pytest
import torch

from hypergraphrewritingengine_b200 import Engine, api
from oracle import pyoracle
from parity import assert_same, norm_gpu, norm_oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    e = Engine(0)
    yield e
    e.close()


def _edges(res, s):
    """The edges of state s as the result stores them."""
    e0, e1 = res.state_edge_off[s: s + 2]
    ends = res.state_vert_off[s] + np.cumsum(res.state_arity[e0:e1].astype(np.int64))
    return [v.tolist() for v in np.split(res.state_verts[res.state_vert_off[s]: ends[-1]],
                                         (ends - res.state_vert_off[s])[:-1])]


def _chain(n):
    return [[i, i + 1] for i in range(1, n)] + [[n, 1]]


# loops, then edges out of the first loops' vertices: the only matches of the rule hold the
# positions p and p + 256
LOOPS = [[i, i] for i in range(1, 257)] + [[i, 1000 + i] for i in range(1, 25)]
CASES = {
    "chain-255": (([[0, 1], [1, 2]], [[0, 1], [1, 2], [2, 0]]), _chain(255), True, 20),
    "chain-256": (([[0, 1], [1, 2]], [[0, 1], [1, 2], [2, 0]]), _chain(256), True, 20),
    "chain-257": (([[0, 1], [1, 2]], [[0, 1], [1, 2], [2, 0]]), _chain(257), True, 20),
    "chain-300": (([[0, 1], [1, 2]], [[2, 0]]), _chain(300), False, 700),
    "chain-520": (([[0, 1], [1, 2]], [[0, 1], [1, 2], [2, 0]]), _chain(520), True, 5),
    "p-and-p+256": (([[0, 0], [0, 1]], [[0, 1], [1, 2]]), LOOPS, False, 0),
    "five-lhs-260": (([[0, 1], [1, 2], [2, 3], [3, 4], [4, 5]], [[0, 5], [5, 6]]), _chain(260), False, 300),
}


@pytest.mark.parametrize("forwarding", [0, 1])
@pytest.mark.parametrize("name", sorted(CASES))
def test_positions_past_a_byte(eng, name, forwarding):
    rule, root, quotient, cap = CASES[name]
    eng.set_option(api.OPT_FORWARDING, forwarding)
    res = eng.evolve([rule], [root], 2, quotient=quotient, max_states=cap)
    eng.set_option(api.OPT_FORWARDING, 0)
    ref = pyoracle.evolve([rule], [root], 2, quotient=quotient, max_states=cap)
    assert_same(norm_gpu(res), norm_oracle(ref), name)
    # a stored state is the one its hash was taken of
    for s in sorted({0, 1, 7, len(res.state_hash) // 2, len(res.state_hash) - 1}):
        if s < len(res.state_hash):
            assert pyoracle.wl_hash(_edges(res, s)) == int(res.state_hash[s]), (name, s)


@pytest.mark.parametrize("rule", [([[0, 1], [0, 2]], [[1, 2]]), ([[0, 1]], [[0, 1], [0, 2]])])
def test_hub_vertex_join_index(eng, rule):
    """A vertex in every edge: its list in the join index ascends (matches in canonical order, as without
    the index), and building it for every unit of work does not cost the square of its degree."""
    n = 150 if len(rule[0]) == 2 else 1500
    star = [[1, k] for k in range(2, n)] + [[1, 1], [2, 1], [1, 2]]
    out, ms = [], []
    for index in (0, 1):
        eng.set_option(api.OPT_JOIN_INDEX, index)
        best = 1e9
        for _ in range(3):
            t = time.perf_counter()
            res = eng.evolve([rule], [star], 1, quotient=False, max_states=3000)
            best = min(best, time.perf_counter() - t)
        out.append(res)
        ms.append(1e3 * best)
    eng.set_option(api.OPT_JOIN_INDEX, 1)
    assert np.array_equal(out[0].events, out[1].events)
    assert np.array_equal(out[0].event_cons, out[1].event_cons)
    assert np.array_equal(out[0].state_hash, out[1].state_hash)
    assert ms[1] < 3 * ms[0] + 2, ms


def test_states_past_4096_edges(eng):
    """Unary edges of one vertex, 3,560 at the start and 15 more a step: 16-bit occurrences in the warp
    hash leave the edge all bits that the arity does not need."""
    steps = 38
    res = eng.evolve([([[0]], [[0]] * 16)], [[[1]] * 3560], steps, quotient=True)
    sizes = [3560 + 15 * d for d in range(steps + 1)]
    assert sizes[-1] > 4096 + 16
    assert [int(h) for h in res.state_hash] == [pyoracle.wl_hash([[1]] * n) for n in sizes]
    assert len(res.events) == sum(sizes[:-1])
    assert len(res.branchial) == 0
    for d in (0, 35, 37, steps):
        assert np.diff(res.state_edge_off)[d] == sizes[d]


def _paths(edges, k):
    """Positions of every path of k edges, in canonical (lexicographic) order."""
    out = {}
    for i, (a, b) in enumerate(edges):
        out.setdefault(a, []).append((i, b))
    found = []

    def walk(v, taken):
        if len(taken) == k:
            found.append(list(taken))
            return
        for i, b in out.get(v, ()):
            if i not in taken:
                walk(b, taken + [i])

    for i, (a, b) in enumerate(edges):
        walk(b, [i])
    return found


@pytest.mark.parametrize("n,vertices,seed", [(48, 9, 1), (100, 25, 2)])
def test_long_slices_of_a_long_rule(eng, n, vertices, seed):
    """More than 20,000 matches of a rule of five left-hand edges: slices longer than the usual list."""
    edges = np.random.default_rng(seed).integers(1, vertices + 1, (n, 2)).tolist()
    want = _paths(edges, 5)
    assert len(want) > 20000
    rule = ([[k, k + 1] for k in range(5)], [[0, 5], [5, 6]])
    eng.set_option(api.OPT_RECORD_BRANCHIAL, 0)
    res = eng.evolve([rule], [edges], 1, quotient=True)
    eng.set_option(api.OPT_RECORD_BRANCHIAL, 1)
    assert np.array_equal(res.event_cons.reshape(-1, 5), np.array(want))


def test_long_slices_of_forwarded_states(eng):
    """90,000 events of 70-edge states, forwarded and joined again: the same arrays."""
    edges = np.random.default_rng(5).integers(1, 31, (70, 2)).tolist()
    rule = ([[0, 1], [1, 2], [2, 3]], [[0, 3], [3, 4]])
    out = []
    for forwarding in (0, 1):
        eng.set_option(api.OPT_FORWARDING, forwarding)
        out.append(eng.evolve([rule], [edges], 2, quotient=True))
    eng.set_option(api.OPT_FORWARDING, 0)
    assert len(out[0].events) > 80000
    for name in ("state_hash", "events", "event_cons", "causal", "branchial"):
        assert np.array_equal(getattr(out[0], name), getattr(out[1], name)), name


def test_hashed_states_past_the_segment_limits_share_the_gpu():
    """hgx_hash_states_noalloc: 64 states of 200 edges, a warp each at once, not one after another."""
    import test_zz_no_alloc as Z
    from hypergraphrewritingengine_b200 import load_library
    states = [np.random.default_rng(k).integers(1, 120, (200, 2)).tolist() for k in range(64)]
    ms = []
    for n in (1, 64):
        dev = torch.device("cuda", 0)
        bufs = [torch.from_numpy(a.view(np.int32 if a.itemsize == 4 else np.int64)).to(dev)
                for a in Z._records(states[:n])]
        out = [torch.empty(n, dtype=torch.int64, device=dev), torch.empty(n, dtype=torch.int32, device=dev)]
        p = [ctypes.c_void_p(t.data_ptr()) for t in bufs + out]
        best = 1e9
        for _ in range(20):
            torch.cuda.synchronize()
            t = time.perf_counter()
            status = load_library().hgx_hash_states_noalloc(
                *p[:4], n, 200, 400, p[4], p[5], ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
            torch.cuda.synchronize()
            best = min(best, time.perf_counter() - t)
            assert status == 0
        assert [int(h) & (2 ** 64 - 1) for h in out[0].tolist()] == [pyoracle.wl_hash(s) for s in states[:n]]
        ms.append(1e3 * best)
    assert ms[1] < 4 * ms[0], ms


@pytest.mark.parametrize("spare", [0, 30])
def test_pairs_of_a_level_past_32_bits(eng, spare):
    """124,950 matches of one state that all hold its one loop: 7.8 billion branchial pairs, an error
    before any is written (of a 52-edge state by the warp's count, of an 82-edge one by the walk)."""
    star = [[1, 1]] + [[1, k] for k in range(2, 53)] + [[100 + 2 * k, 101 + 2 * k] for k in range(spare)]
    rule = ([[0, 0], [0, 1], [0, 2], [0, 3]], [[1, 2]])
    with pytest.raises(api.HgxError, match="branchial pairs") as err:
        eng.evolve([rule], [star], 1, quotient=True)
    assert err.value.status == api.HGX_ERR_CAPACITY
    eng.set_option(api.OPT_RECORD_BRANCHIAL, 0)   # without them the level is an ordinary one
    res = eng.evolve([rule], [star], 1, quotient=True)
    eng.set_option(api.OPT_RECORD_BRANCHIAL, 1)
    assert len(res.events) == 51 * 50 * 49
    small = eng.evolve([rule], [star[:8]], 1, quotient=True)   # and the engine goes on
    assert len(small.branchial) == 210 * 209 // 2


def test_events_of_a_level_past_32_bits(eng):
    """301 states of 14,295,960 matches each: more events than 32-bit ids, an error before any is built."""
    roots = [[[r, 1000 + 63 * r + k] for k in range(63)] for r in range(301)]
    with pytest.raises(api.HgxError, match="32-bit id space exhausted") as err:
        eng.evolve([([[0, 1], [0, 2], [0, 3], [0, 4]], [[1, 2]])], roots, 1, quotient=True)
    assert err.value.status == api.HGX_ERR_CAPACITY
    assert len(eng.evolve([([[0, 1], [0, 2]], [[1, 2]])], [roots[0]], 1).events) == 63 * 62
