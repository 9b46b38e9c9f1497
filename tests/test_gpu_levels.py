"""Small levels in one cooperative launch against the ordinary level pipeline.

Per-stage timing (HGX_OPT_TIMING = 1) turns the launch off, so the same call runs on both paths;
every result array must be equal, ids and order included. The cases sit at the edges of the
launch's rule: levels just below and above its event limit, states around 63 / 64 edges (branchial
masks, lane walks against index walks and the join index), several rules and roots, unary and mixed
arities, a deleting rule, caps out of and within reach, evolutions that stop in different levels of
one batch, and levels run one per call by the serving steps.
"""
import numpy as np
import pytest

import cases
from hypergraphrewritingengine_b200 import Engine, api
from hypergraphrewritingengine_b200 import workloads as W

pytestmark = pytest.mark.gpu

ARRAYS = ("state_hash", "state_depth", "events", "causal", "branchial", "event_cons_off",
          "event_cons", "event_prod", "state_edge_off", "state_edge_ids", "state_arity",
          "state_vert_off", "state_verts", "event_signature")


def same_arrays(a, b, what):
    for name in ARRAYS:
        assert np.array_equal(getattr(a, name), getattr(b, name)), (what, name)
    assert (a.num_classes, a.num_canonical_events, a.truncated) == \
        (b.num_classes, b.num_canonical_events, b.truncated), what


@pytest.fixture(scope="module")
def engines():
    both = Engine(0), Engine(0)
    both[1].set_option(api.OPT_TIMING, 1)
    yield both
    for e in both:
        e.close()


def _chain(n):
    return [[i, i + 1] for i in range(1, n)] + [[n, 1]]


GROW = [([[0, 1], [1, 2]], [[0, 1], [1, 2], [2, 0]])]
SINGLE = {name: (rules, roots, steps, False, 0) for name, rules, roots, steps in cases.all_full_cases()
          if name.startswith("edge-") or name.startswith("corpus-")}
SINGLE.update({
    "wpp-7": ([cases.C2_RULE], [cases.C2_INIT], 7, True, 0),            # past the event limit
    "wpp-full-4": ([cases.C2_RULE], [cases.C2_INIT], 4, False, 0),
    "ternary-5": ([cases.C3_RULE], [cases.C3_INIT], 5, True, 0),
    "cap-far": ([cases.C2_RULE], [cases.C2_INIT], 5, True, 100000),
    "cap-near": ([cases.C2_RULE], [cases.C2_INIT], 6, True, 700),
    "cap-full": ([cases.C1_RULE], [cases.C1_INIT], 5, False, 900),
    "edges-62": (GROW, [_chain(62)], 2, True, 0),
    "edges-63": (GROW, [_chain(63)], 2, True, 0),
    "edges-64": (GROW, [_chain(64)], 2, True, 0),
    "edges-97": (GROW, [_chain(97)], 2, True, 0),
    "edges-97-roots": (GROW, [_chain(97), _chain(40), _chain(97)], 1, True, 0),
    "no-match": ([([[0, 1, 2]], [[0, 1]])], [_chain(3)], 3, True, 0),
    "long-lhs": ([([[0, 1], [1, 2], [2, 3], [3, 4], [4, 5]], [[0, 5], [5, 6]])], [_chain(12)], 3, True, 0),
    # counting stops: enumerated matches of one state, and those of a state past 64 edges
    "long-lhs-1944": ([([[0, 1], [1, 2], [2, 3], [3, 4], [4, 5]], [[0, 5]])],
                      [[[i, i + 1] for i in range(1, 13) for _ in range(3)]], 1, True, 0),
    "star-19460": ([([[0, 1], [0, 2]], [[1, 2]])], [[[1, i] for i in range(2, 142)]], 1, True, 0),
    "20-levels": ([([[0, 1]], [[1, 0]])], [_chain(5)], 20, True, 0),    # more levels than one launch takes
})


# Cases with no level inside the launch, and those with some.
LEFT = {"long-lhs-1944", "star-19460"}
PARTLY = {"cap-full", "cap-near", "ternary-5", "wpp-7", "wpp-full-4"}


@pytest.mark.parametrize("reduce,keys", [(False, 0), (True, 3)])
@pytest.mark.parametrize("name", sorted(SINGLE))
def test_single_evolutions(engines, name, reduce, keys):
    rules, roots, steps, quotient, cap = SINGLE[name]
    out, launches = [], []
    for eng in engines:
        eng.set_option(api.OPT_TRANSITIVE_REDUCTION, reduce)
        eng.set_option(api.OPT_EVENT_SIGNATURE_KEYS, keys)
        out.append(eng.evolve(rules, roots, steps, quotient=quotient, max_states=cap))
        launches.append(eng.stage_times()[1])
        eng.set_option(api.OPT_TRANSITIVE_REDUCTION, False)
        eng.set_option(api.OPT_EVENT_SIGNATURE_KEYS, 0)
    same_arrays(*out, name)
    # that the launch did run: a level of the ordinary pipeline is at least ten launches
    if name in LEFT:
        assert launches[0] > launches[1], launches
    elif name in PARTLY:
        assert launches[0] < launches[1] - 20, launches
    else:
        assert launches[0] < 10, launches


@pytest.mark.parametrize("n,cap", [(1, 50), (37, 200), (300, 4096)])
def test_batches(engines, n, cap):
    evs = [W.random_evolution(i, seed=71 + n, max_states=cap, edges_hi=40, steps_lo=0, steps_hi=4)
           for i in range(n)]
    for i, (a, b) in enumerate(zip(*(eng.evolve_batch(evs) for eng in engines))):
        same_arrays(a, b, i)
    if n < 300:   # (300 start with more events than a level of the launch takes)
        assert engines[0].stage_times()[1] < engines[1].stage_times()[1]


def test_record_options_and_serving_steps(engines):
    evs = [W.random_evolution(i, seed=5, max_states=300, edges_hi=30, steps_hi=5) for i in range(12)]
    for causal, branchial in ((False, True), (True, False)):
        out = []
        for eng in engines:
            eng.set_option(api.OPT_RECORD_CAUSAL, causal)
            eng.set_option(api.OPT_RECORD_BRANCHIAL, branchial)
            eng.serve_reset()
            jobs, keep = eng.make_jobs(evs)
            ids = eng.serve_admit_batch(jobs, 7)
            got, more = {}, 7
            while len(got) < len(evs):
                for k, r in zip(*(lambda d: (d, eng.serve_collect_batch(d)))(eng.serve_take_finished())):
                    got[k] = r
                if more < len(evs):     # one more request between the levels of the others
                    ids.append(eng.serve_admit(jobs[more]))
                    more += 1
                eng.serve_step()
            out.append([got[i] for i in ids])
            eng.set_option(api.OPT_RECORD_CAUSAL, True)
            eng.set_option(api.OPT_RECORD_BRANCHIAL, True)
        for i, (a, b) in enumerate(zip(*out)):
            same_arrays(a, b, (causal, branchial, i))


@pytest.mark.parametrize("n", [31, 33, 319, 321, 640, 641, 700])
def test_hub_vertex_hashes(engines, n):
    """One vertex in n edges: its neighbour words pass the registers' 32 and the buffer's 640 (an
    arity-3 hub twice as early), its occurrences the buffer of a mixed-arity state's first colours."""
    from oracle import pyoracle
    star = [[1, i + 2] for i in range(n)]
    roots = [star, [e + [e[1] % 7 + 2] for e in star], star + [[1], [1], [2, 3, 1]],
             [[1]] * n + star[: n // 2], [[1, 1]] * (n // 2) + [[1, 2]]]
    res = engines[0].evolve([([[0, 1]], [[0, 1]])], roots, 0, quotient=False)
    assert [int(h) for h in res.state_hash] == [pyoracle.wl_hash(r) for r in roots]


@pytest.mark.parametrize("arity,n_lhs", [(2, 2), (3, 2), (2, 3), (2, 5)])
def test_large_state_joins(engines, arity, n_lhs):
    """States of 65-130 edges: index walks (rules of up to four left-hand edges) and the warp join
    against the oracle, with and without the join index."""
    from oracle import pyoracle
    rng = W.SplitMix64(41 + arity + n_lhs)
    lhs = [[k] + [k + 1] * (arity - 1) if k % 2 else [k + 1] + [k] * (arity - 1) for k in range(n_lhs)]
    rule = (lhs, [[n_lhs, 0] + [n_lhs + 1] * (arity - 2), [n_lhs + 1] * arity])
    for edges in (65, 97, 130):
        root = W.random_hypergraph(rng, edges, arity) + [[5] * arity, [6] * arity]
        ref = pyoracle.evolve([rule], [root], 2, quotient=True, max_states=60)
        want = pyoracle.normalize(ref["state_hash"], ref["events"], ref["causal"], ref["branchial"])
        for index in (1, 0):
            engines[0].set_option(api.OPT_JOIN_INDEX, index)
            res = engines[0].evolve([rule], [root], 2, quotient=True, max_states=60)
            got = pyoracle.normalize(res.state_hash, res.events, res.causal, res.branchial)
            for k in want:
                assert np.array_equal(got[k], want[k]), (edges, index, k)
        engines[0].set_option(api.OPT_JOIN_INDEX, 1)


def test_long_right_hand_sides(engines):
    """Right-hand sides of more than 32 positions (15 binary edges and a ternary one) in the lane and
    warp kernels, against the oracle."""
    from oracle import pyoracle
    rhs = [[k % 3, (k + 1) % 4] for k in range(15)] + [[0, 1, 2]]
    rules = [([[0, 1], [1, 2]], rhs), ([[0, 1, 2]], [[0, 1], [1, 2]])]
    roots = [[[1, 2], [2, 3], [3, 1]]]
    ref = pyoracle.evolve(rules, roots, 2, quotient=True)
    want = pyoracle.normalize(ref["state_hash"], ref["events"], ref["causal"], ref["branchial"])
    for eng in engines:
        res = eng.evolve(rules, roots, 2, quotient=True)
        got = pyoracle.normalize(res.state_hash, res.events, res.causal, res.branchial)
        for k in want:
            assert np.array_equal(got[k], want[k]), k


def test_noalloc_states_at_the_segment_limits():
    """hgx_hash_states_noalloc on both of its kernels: 31-33 vertices, 63-65 edges, one arity of 1 to 4
    and mixed ones, components, a hub, and labels at the ends of their range."""
    import test_zz_no_alloc as Z
    from hypergraphrewritingengine_b200 import load_library
    from oracle import pyoracle
    states = []
    for arity in (1, 2, 3, 4):
        for nv in (1, 2, 16, 17, 31, 32, 33):
            for ne in (1, 2, 31, 32, 33, 63, 64, 65):
                states.append([[(k * (q + 1) + q) % nv for q in range(arity)] for k in range(ne)])
    states += [[[1, 2], [2, 3, 4]], [[1, 2], [3, 4], [5, 6]], [[0, 2], [3, 0]], [[0xFFFFFFFE, 5], [5, 0xFFFFFFFE]],
               [[7, k] for k in range(8, 39)], [[7, k, 7] for k in range(8, 39)], [[3, 3], [3, 3], [4, 3]]]
    h, cls = Z._noalloc(load_library(), states)
    want = [pyoracle.wl_hash(s) for s in states]
    assert [int(x) for x in h] == want
    assert [int(c) for c in cls] == [want.index(x) for x in want]


@pytest.mark.parametrize("barrier", [1, 2, 5, 6, 9, 13, 14])
def test_a_barrier_that_closes_leaves_the_level_to_the_ordinary_pipeline(engines, barrier):
    """A level's first two barriers run out: the launch ends there for every block -- also for one that
    is still on its way out of the barrier before (5, 9, 13: the first of a later level) -- and the
    level is run again over the tables it has partly filled."""
    rules, roots, steps, quotient, cap = SINGLE["ternary-5"]
    want = engines[1].evolve(rules, roots, steps, quotient=quotient, max_states=cap)
    engines[0].evolve(rules, roots, steps, quotient=quotient, max_states=cap)
    usual = engines[0].stage_times()[1]
    engines[0].set_option(api.OPT_HASTY_BARRIER, barrier)
    try:
        for _ in range(20):
            same_arrays(engines[0].evolve(rules, roots, steps, quotient=quotient, max_states=cap), want, barrier)
            assert engines[0].stage_times()[1] > usual   # (launches: the repeated level's)
    finally:
        engines[0].set_option(api.OPT_HASTY_BARRIER, 0)


@pytest.mark.parametrize("barrier", [3, 4, 8])
def test_a_barrier_that_closes_after_the_expansion_fails_the_call(engines, barrier):
    rules, roots, steps, quotient, cap = SINGLE["ternary-5"]
    want = engines[1].evolve(rules, roots, steps, quotient=quotient, max_states=cap)
    engines[0].set_option(api.OPT_HASTY_BARRIER, barrier)
    try:
        with pytest.raises(api.HgxError) as err:
            engines[0].evolve(rules, roots, steps, quotient=quotient, max_states=cap)
        assert err.value.status == api.HGX_ERR_INTERNAL
    finally:
        engines[0].set_option(api.OPT_HASTY_BARRIER, 0)
    same_arrays(engines[0].evolve(rules, roots, steps, quotient=quotient, max_states=cap), want, barrier)


def test_one_state_of_many_matches_reserves_the_pairs_it_has():
    """14,280 matches of one state: 102 million possible pairs, of which 3.4 million share an edge."""
    eng = Engine(0)
    star = [[1, k] for k in range(2, 122)]
    res = eng.evolve([([[0, 1], [0, 2]], [[1, 2]])], [star], 1, quotient=False)
    assert len(res.events) == 120 * 119
    assert len(res.branchial) == 14280 * (4 * 118 + 1) // 2   # (each shares an edge with 4 * 118 + 1 others)
    assert eng.device_bytes() < 200 << 20
    eng.close()


def test_two_engines_on_two_threads():
    """Two cooperative launches at a time, each on its own engine's stream: every result as alone."""
    import threading
    names = ["wpp-full-4", "ternary-5", "edges-97", "edge-multi-root-3", "long-lhs"]
    both = Engine(0), Engine(0)

    def call(eng, name):
        rules, roots, steps, quotient, cap = SINGLE[name]
        return eng.evolve(rules, roots, steps, quotient=quotient, max_states=cap)

    alone = {name: call(both[0], name) for name in names}
    failed = []

    def work(k):
        try:
            for i in range(60):
                name = names[(i + k * 2) % len(names)]
                same_arrays(call(both[k], name), alone[name], (k, i, name))
        except BaseException as e:   # (reported by the main thread)
            failed.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for e in both:
        e.close()
    assert not failed, failed
