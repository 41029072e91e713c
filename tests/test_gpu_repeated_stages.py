"""Stages run again, out of the chain's order or on nothing: the linking stages after a caller's links, a batch of no
events, connectivity with another cut, and the times of a stage that runs again by itself."""
import numpy as np
import pytest

from trax_gb300 import events

pytestmark = pytest.mark.gpu


def _links_between_levels(level, n_links, down, seed):
    """Links without a cycle (along a random order of the triplets) between triplets of different levels, upwards only
    or in both directions, by basis, each once."""
    rng = np.random.default_rng(seed)
    n = level.size
    rank = rng.permutation(n)
    b, f = rng.integers(0, n, (2, 8 * n_links))
    keep = (rank[b] < rank[f]) & (level[b] != level[f]) if down else level[b] < level[f]
    return np.unique(np.stack([b[keep], f[keep]], axis=1), axis=0)[:n_links].T


def _ca_by_levels(level, b, f, pt):
    """The automaton swept once over the levels: a triplet's state is one above its highest basis, the best basis the
    one of the state below with the least pt difference, the lowest index of several.  A link against the levels can
    leave a state without such a base: the track ends there, its further places (-1 here) hold nothing."""
    n = level.size
    bases = [[] for _ in range(n)]
    for i, j in zip(b, f):
        bases[j].append(i)
    state = np.ones(n, np.int64)
    for lv in range(1, int(level.max()) + 1):
        new = {t: 1 + max(state[bases[t]]) for t in np.nonzero(level == lv)[0] if bases[t]}
        for t, s in new.items():
            state[t] = s
    best, is_best = np.full(n, -1), np.zeros(n, bool)
    for t in range(n):
        ok = [k for k in bases[t] if state[k] + 1 == state[t]]
        if ok:
            best[t] = min(ok, key=lambda k: (abs(pt[k] - pt[t]), k))
            is_best[best[t]] = True
    tracks, offsets = [], [0]
    for t in range(n):
        k, length = t, 0 if is_best[t] else state[t]
        for _ in range(length):
            tracks.append(k)
            k = best[k] if k >= 0 else -1
        offsets.append(len(tracks))
    return state, np.array(tracks), np.array(offsets)


@pytest.mark.parametrize("down", [False, True])
@pytest.mark.parametrize("graph", [False, True])
def test_ca_stage_on_a_callers_links(trax_lib, graph, down):
    """trax_cellular_automaton right after trax_cellular_automaton_on takes that call's links and pt, which may cross
    events and go against the levels: one sweep over the levels of all events."""
    batch = events.generate(2, n_events=4)
    with trax_lib.Context(0) as ctx:
        ctx.upload(batch)
        ctx.seed_batch(use_graph=graph)
        first = ctx.results()
        level = batch.layer[first["perm"]][first["trip_h1"]].astype(np.int64) - 1
        event = batch.event[first["perm"]][first["trip_h1"]]
        pt = np.random.default_rng(1).choice(np.float32([10.0, 20.0, 33.25, 50.0]), level.size)
        b, f = _links_between_levels(level, 3 * level.size // 2, down, seed=2)
        assert (event[b] != event[f]).any() and (not down or (level[b] > level[f]).any())
        want = _ca_by_levels(level, b, f, pt)
        by_caller = ctx.cellular_automaton_on(b, f, pt)
        for run in range(2):
            ctx.cellular_automaton()
            got = ctx.tracks()
            for w, g, name in zip(want, got, ("states", "tracks", "offsets")):
                assert g.shape == w.shape and np.array_equal(g[w >= 0], w[w >= 0]), (run, name)
        if not down:  # upwards the sweep is the reference's iteration
            assert all(np.array_equal(g, w) for g, w in zip(got, by_caller))
        # the chain's own links again
        assert ctx.connectivity(batch.d_eta_cut) == first["link_basis"].size
        ctx.circle_fit()
        ctx.cellular_automaton()
        again = ctx.results()
    for k, v in first.items():
        assert np.array_equal(v, again[k]), k


@pytest.mark.parametrize("linking", [True, False])
@pytest.mark.parametrize("graph", [False, True])
def test_batch_of_no_events(trax_lib, graph, linking):
    """No events (an empty shard) run in both modes and give nothing, before and after a batch that gives something."""
    some = events.generate(2, n_events=2)
    none = some.subset([])
    with trax_lib.Context(0) as ctx:
        ctx.upload(none)
        counts = []
        for batch in (none, none, some, none, some):
            ctx.upload_hits(batch)
            st = ctx.seed_batch(use_graph=graph, run_linking=linking)
            counts.append((st.n_pairs, st.n_candidates, st.n_triplets, st.n_links, st.n_track_entries))
            h1, _, _, offsets = ctx.triplets()
            assert h1.size == st.n_triplets and offsets[-1] == max(st.n_triplets, 1) - 1
            if linking:
                assert ctx.tracks()[1].size == st.n_track_entries
    assert counts[0] == counts[1] == counts[3] == (0,) * 5
    assert counts[2] == counts[4] and counts[2][2] > 0 and (counts[2][3] > 0) == linking


@pytest.mark.parametrize("graph", [False, True])
def test_tracks_after_connectivity_again(trax_lib, graph):
    """Connectivity run again leaves no earlier automaton's tracks: none with a cut that links nothing (the caller's
    arrays stay as they are), an error until the automaton has run with one that links."""
    batch = events.generate(2, n_events=3)
    with trax_lib.Context(0) as ctx:
        ctx.upload(batch)
        ctx.seed_batch(use_graph=graph)
        first = ctx.results()
        assert first["tracks"].size > 0

        def untouched():
            n = first["trip_h1"].size
            out = [np.full(k, 7, np.uint32) for k in (n, first["tracks"].size, n + 1)]
            ctx.tracks(out=out)
            return all((v == 7).all() for v in out)

        assert ctx.connectivity(0.0) == 0
        assert untouched()
        ctx.circle_fit()
        assert ctx.cellular_automaton() == 0
        assert untouched()
        assert ctx.connectivity(batch.d_eta_cut) == first["link_basis"].size
        with pytest.raises(trax_lib.TraxError) as e:
            ctx.tracks()
        assert e.value.code == 6
        ctx.circle_fit()
        ctx.cellular_automaton()
        again = ctx.results()
    for k, v in first.items():
        assert np.array_equal(v, again[k]), k


def test_circle_fit_when_connectivity_linked_nothing(trax_lib):
    """trax_circle_fit fits the connectable triplets of the last connectivity: none, when that linked nothing, also after
    trax_cellular_automaton_on gave the context links of the caller's."""
    batch = events.generate(2, n_events=3)
    with trax_lib.Context(0) as ctx:
        ctx.upload(batch)
        n = ctx.seed_batch(use_graph=False).n_triplets
        assert (ctx.eta_pt()[1] > 0).any()
        assert ctx.connectivity(0.0) == 0
        ctx.cellular_automaton_on([0, 1], [n - 1, n - 1], np.ones(n, np.float32))
        ctx.circle_fit()
        assert (ctx.eta_pt()[1] == 0).all()


def test_times_of_a_stage_run_again(trax_lib):
    """A stage that runs again by itself has its new time and leaves the others theirs; every timed kernel lies inside
    its stage."""
    inside = {"grid": ["grid_build"], "pairs": ["pair_count", "pair_store"],
              "predict": ["predict_count", "predict_store"], "filter": ["filter", "filter_store"],
              "connectivity": ["connectivity_count", "connectivity_store"]}
    batch = events.generate(2, n_events=3)
    with trax_lib.Context(0) as ctx:
        ctx.upload(batch)
        ctx.seed_batch(use_graph=True)
        ctx.seed_batch(use_graph=True)
        stage, kernel = ctx.timings()
        for s, ks in inside.items():
            assert 0 < sum(kernel[k] for k in ks) <= stage[s] + 1e-6, s
        ctx.seed_batch(use_graph=False)
        before, kernel = ctx.timings()
        for s, ks in inside.items():
            assert 0 < sum(kernel[k] for k in ks) <= before[s] + 1e-6, s
        for again, run in (("connectivity", lambda: ctx.connectivity(batch.d_eta_cut)), ("pairs", ctx.pair_gen)):
            run()
            after, _ = ctx.timings()
            assert 0 < after[again] < 1e3
            assert {s: t for s, t in after.items() if s != again} == {s: t for s, t in before.items() if s != again}
            before = after
