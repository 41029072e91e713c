"""Launch structure of the chain: time marks."""
import dataclasses

import numpy as np
import pytest

from trax_gb300 import events

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [True, False])
def test_time_marks_fit_the_device_time(trax_lib, graph):
    """Every stage and timed kernel of a run has a time, kernels lie inside their stages, and the stages together
    stay within the device time of the whole run (CUDA events around it; 10 us for the two clocks)."""
    batch = events.generate(1, n_events=8)
    with trax_lib.Context(0) as ctx:
        ctx.upload(batch)
        for _ in range(3):
            st = ctx.seed_batch(use_graph=graph)
        stage, kernel = ctx.timings()
    assert all(v > 0 for v in stage.values()) and all(v > 0 for v in kernel.values())
    assert sum(stage.values()) <= st.device_ms + 0.01
    assert kernel["pair_count"] + kernel["pair_store"] <= stage["pairs"] + 1e-6
    assert kernel["filter"] + kernel["filter_store"] <= stage["filter"] + 1e-6
    assert np.isclose(kernel["grid_build"], stage["grid"], rtol=0, atol=stage["grid"])


@pytest.mark.parametrize("n_events", [1, 8191, 8192, 32767, 32768])
def test_segment_scan_sizes(trax_lib, n_events):
    """Segments in one CTA's steps (8192 each, up to 32767) and past its limit: copies of a few small events give the
    copies of their results."""
    few = events.generate(0, n_events=7)
    batch = few.subset([e % 7 for e in range(n_events)])
    with trax_lib.Context(0) as ctx:
        ctx.upload(few)
        ctx.seed_batch(use_graph=False, run_linking=False)
        _, pair_offsets = ctx.pairs()
        _, cand_offsets = ctx.candidates()
        h1, _, h3, _ = ctx.triplets()
    want = [np.concatenate([[0], np.cumsum(np.diff(o.astype(np.int64))[np.arange(n_events) % 7])])
            for o in (pair_offsets, cand_offsets)]
    starts = batch.event_offsets
    with trax_lib.Context(0) as ctx:
        ctx.upload(batch)
        for graph in (False, True):
            ctx.seed_batch(use_graph=graph, run_linking=False)
            p, po = ctx.pairs()
            c, co = ctx.candidates()
            assert np.array_equal(po, want[0]) and np.array_equal(co, want[1])
            assert p.shape[0] == po[-1] and c.shape[0] == co[-1]
            k1, _, k3, off = ctx.triplets()
            # the first copy of event 0 comes out as alone, and every hit lies in its own event
            e = batch.event[k1]
            assert np.array_equal(e, batch.event[k3]) and np.all(np.diff(e.astype(np.int64)) >= 0)
            first = few.event[h1] == 0
            assert np.array_equal(k1[e == 0], h1[first]) and np.array_equal(k3[e == 0], h3[first])
            last = n_events - 1
            alone = few.event[h1] == last % 7
            shift = int(starts[last]) - int(few.event_offsets[last % 7])
            assert np.array_equal(k1[e == last], h1[alone] + shift)


@pytest.mark.parametrize("where", [(0, 1, 2), (5, 40, 299), (0, 150, 298), (297, 298, 299)])
@pytest.mark.parametrize("graph", [True, False])
def test_segments_between_empty_events(trax_lib, oracle_lib, where, graph):
    """Triplet segments and offsets with runs of empty segments before, between and after the ones that hold triplets
    (gaps shorter and longer than a warp), and the CA's event blocks without triplets: every array as the oracle's."""
    few = events.generate(1, n_events=3)
    layer_hits = np.zeros((300, few.n_layers), dtype=np.uint32)
    layer_hits[list(where)] = few.layer_hits
    cols = {k: getattr(few, k) for k in ("x", "y", "z", "layer", "det_id", "hit_id")}
    cols["event"] = np.asarray(where, dtype=np.uint32)[few.event]
    batch = events._assemble(cols, layer_hits, few)
    want = oracle_lib.run(batch)[0]
    with trax_lib.Context(0) as ctx:
        ctx.upload(batch)
        ctx.seed_batch(use_graph=graph)
        got = ctx.results()
    for name in ("pair_offsets", "cand_offsets", "trip_offsets", "trip_h1", "trip_h2", "trip_h3", "link_basis",
                 "link_follower", "connectable", "non_connectable", "ca_states", "tracks", "track_offsets"):
        assert np.array_equal(got[name], want[name]), name


def test_linking_after_a_callers_links(trax_lib):
    """trax_cellular_automaton_on takes the incoming-link lists for its own links; the chain's linking stages run
    again on the context give what they gave before."""
    batch = events.generate(1, n_events=6)
    with trax_lib.Context(0) as ctx:
        ctx.upload(batch)
        ctx.seed_batch(use_graph=False)
        first = ctx.results()
        n = first["trip_h1"].size
        ctx.cellular_automaton_on([0, 1], [n - 1, n - 1], np.ones(n, np.float32))
        assert ctx.connectivity(batch.d_eta_cut) == first["link_basis"].size
        ctx.circle_fit()
        ctx.cellular_automaton()
        again = ctx.results()
        b, f = first["link_basis"], first["link_follower"]
        by_caller = ctx.cellular_automaton_on(b, f, first["pt"])  # the chain's links as a caller's
    for k, v in first.items():
        assert np.array_equal(v, again[k]), k
    for v, k in zip(by_caller, ("ca_states", "tracks", "track_offsets")):
        assert np.array_equal(v, first[k]), k


@pytest.mark.parametrize("n_z, n_phi", [(80, 256), (4, 8), (1, 1), (3, 40)])
def test_mask_walk_range_lengths(trax_lib, oracle_lib, n_z, n_phi):
    """The prediction's walk by masks (8 or more captured candidates) over visit ranges from none to far more than
    the 32 hits of a mask, the last layer's hits at the end of the hit arrays included: every array as the oracle's."""
    batch = events.generate(1, n_events=5)
    batch.n_z, batch.n_phi = n_z, n_phi
    want = oracle_lib.run(batch)[0]
    with trax_lib.Context(0) as ctx:
        ctx.upload(batch)
        for slots in (16, 32, 8, 4):
            ctx.set_candidate_slots(slots)
            ctx.seed_batch(use_graph=False)
            got = ctx.results()
            for name in ("pairs", "cands", "cand_offsets", "trip_h1", "trip_h2", "trip_h3"):
                assert np.array_equal(got[name], want[name]), (slots, name)


def test_one_graph_serves_a_stream_of_unequal_batches(trax_lib, oracle_lib):
    """Groups of one shape replay one captured graph whatever their number of hits, as long as they fit: more hits than
    the captured buffers, a larger layer than the captured grid layout or more pairs than the capacities capture anew.
    Every group's results are the oracle's."""
    groups = [events.generate(1, n_events=6, seed=s) for s in (3, 4, 5)]
    dense = events.generate_workload(dataclasses.replace(events.workload(1, 6), n_tracks=420), seed=6)
    want = [oracle_lib.run(b)[0] for b in groups + [dense]]
    names = ("pairs", "cands", "trip_offsets", "trip_h1", "trip_h3", "link_basis", "connectable", "tracks")
    with trax_lib.Context(0) as ctx:
        ctx.upload(groups[0])
        captures = []
        for k in (0, 1, 2, 0, 3, 1, 2, 3):
            b = (groups + [dense])[k]
            ctx.upload_hits(b)
            captures.append(ctx.seed_batch(use_graph=True).graph_captures)
            got = ctx.results()
            for name in names:
                assert np.array_equal(got[name], want[k][name]), (k, name)
    assert captures[0] == 1 and captures[3] == 0 and captures[4] >= 1
    assert captures[5:] == [0, 0, 0]  # the dense group's graph holds the others too


@pytest.mark.parametrize("n", [1, 31, 255, 256, 257, 1025])
def test_fit_block_edges(trax_lib, align_ref, n):
    """The fit's sums over n rows (lanes, warps and blocks that are partly empty) against the FP64 reference, the error
    relative to the sum of the rows' magnitudes: 5e-4 (hit gradients of single rows are within 3e-4)."""
    batch = events.generate(4, n_events=2, seed=11)
    batch.n_z, batch.n_phi = 50, 128
    shifts = np.random.default_rng(n).normal(0, 1, (batch.n_layers, 3)) * [0.003, 0.003, 2e-5]
    sigma_tip = [0.01 + 0.01 * k for k in range(len(batch.lts))]
    with trax_lib.Context(0) as ctx:
        ctx.upload(batch)
        ctx.seed_batch(use_graph=False, run_linking=False)
        h1, h2, h3, _ = ctx.triplets()
        perm = ctx.hit_perm().astype(np.int64)
        ids = batch.hit_id[perm]
        good = np.nonzero((ids[h1] != 0) & (ids[h1] == ids[h2]) & (ids[h2] == ids[h3]))[0]
        pick = good[np.linspace(0, good.size - 1, n).astype(np.int64)]
        a, b, c = (perm[h[pick]] for h in (h1, h2, h3))
        key = batch.event[a].astype(np.int64) * 16 + batch.layer[a]
        o = np.argsort(key, kind="stable")
        a, b, c = a[o], b[o], c[o]
        ctx.set_tracklets(a, b, c)
        assert ctx.fit_prepare(sigma_z=0.002, sigma_tip=sigma_tip, truth_only=True) == n
        chi2, grad, _ = ctx.fit_backward(shifts)
        chi2_f, params = ctx.fit_forward(shifts, params=True)
    sig = np.asarray(sigma_tip)[batch.layer[a] - 1]
    args = (batch.x, batch.y, batch.z, batch.layer)
    want, want_grad, _ = align_ref.loss_and_grad(*args, a, b, c, np.ones(n), shifts, sig, 0.002)
    size = sum(np.abs(align_ref.loss_and_grad(*args, a[k:k + 1], b[k:k + 1], c[k:k + 1], np.ones(1), shifts,
                                              sig[k:k + 1], 0.002)[1]) for k in range(n))
    assert abs(chi2 - want) <= 1e-4 * want and chi2_f == pytest.approx(chi2, rel=1e-12)
    assert np.all(np.abs(grad - want_grad) <= 5e-4 * size.max(axis=0))
    assert params.shape == (n, 4) and np.isfinite(params).all()


@pytest.mark.parametrize("tasks", [0, 36000, 120000])
def test_pair_lanes_on_degenerate_windows(trax_lib, oracle_lib, tasks):
    """The pair kernels with 8, 4 and 1 lanes per outer hit (by the number of outer hits) on the degenerate batch's
    windows (NaN, infinite, wider than 2 pi, on cell edges), repeated to reach that number: every copy's pairs are the
    oracle's, sentinels included."""
    from tests.test_oracle_kats import degenerate_batch
    few = degenerate_batch()
    per = sum(int(few.layer_hits[:, lt.layer2 - 1].sum()) for lt in few.lts)
    copies = tasks // per + 1
    batch = few.subset(list(range(few.n_events)) * copies)
    want = oracle_lib.run(few)[0]["pairs"].reshape(-1, 2).astype(np.int64)
    with trax_lib.Context(0) as ctx:
        ctx.upload(batch)
        ctx.grid_build()
        ctx.pair_gen()
        p, off = ctx.pairs()
        st = ctx.stats()
    assert p.shape[0] == copies * want.shape[0] and off[-1] == p.shape[0]
    shift = np.repeat(np.arange(copies) * few.n_hits, want.shape[0])[:, None]
    p = p.astype(np.int64)
    p[p != 0xFFFFFFFF] -= np.broadcast_to(shift, p.shape)[p != 0xFFFFFFFF]
    assert np.array_equal(p, np.tile(want, (copies, 1)))
    assert st.n_pair_sentinels == copies * int((want[:, 0] == 0xFFFFFFFF).sum())


@pytest.mark.parametrize("middle", [(2, 3, 4), (3, 3, 4), (4, 3, 4)])
def test_links_with_and_without_shared_second_layers(trax_lib, oracle_lib, middle):
    """Followers are looked up by the run of triplets with their second hit unless a layer is the second of two layer
    triplets; both give the oracle's links, on a context that had other batches' runs before."""
    lts = events.layer_triplets([1, 2, 3])
    lts = [dataclasses.replace(lt, layer2=m, layer3=max(lt.layer3, m + 1)) for lt, m in zip(lts, middle)]
    batches = [dataclasses.replace(events.generate(2, n_events=n, seed=n), lts=lts) for n in (4, 3)]
    with trax_lib.Context(0) as ctx:
        for b in batches:
            want = oracle_lib.run(b)[0]
            ctx.upload(b)
            ctx.seed_batch(use_graph=False)
            got = ctx.results()
            assert want["link_basis"].size > 0
            for name in ("trip_h2", "link_basis", "link_follower", "connectable", "ca_states", "tracks"):
                assert np.array_equal(got[name], want[name]), name


@pytest.mark.parametrize("fine", [0, 8])
@pytest.mark.parametrize("slots", [16, 32])
def test_candidates_copied_by_output(trax_lib, oracle_lib, slots, fine):
    """The store pass that takes a warp's candidates one per lane: warps whose pairs have from no to far more candidates
    than slots side by side, and a last warp that is not full."""
    lts = [dataclasses.replace(lt, sigma_phi=1.0, sigma_z=5.0) for lt in events.layer_triplets([1])]
    batch = events.generate_workload(dataclasses.replace(events.workload(1, 3), n_tracks=300, lts=lts), seed=8)
    want = oracle_lib.run(batch, links="none")[0]
    per = np.bincount(want["cands"].reshape(-1, 2)[:, 0])
    assert (per == 0).any() and (per > slots).any() and ((per > 0) & (per <= slots)).any()
    assert (want["pairs"].size // 2) % 32
    with trax_lib.Context(0) as ctx:
        ctx.set_candidate_slots(slots)
        ctx.set_fine_rows(fine)
        ctx.upload(batch)
        for graph in (False, True):
            ctx.seed_batch(use_graph=graph, run_linking=False)
            assert np.array_equal(ctx.candidates()[0].ravel(), want["cands"]), graph
            assert ctx.stats().n_candidate_sentinels == want["stats_dict"]["cand_undefined_slots"]


@pytest.mark.parametrize("n", [1, 4096, 4097, 8191, 8192, 8193, 16383, 16384, 16385, 20481])
def test_scan_by_one_block_and_by_tiles(trax_lib, n):
    """Sizes around one tile, around the tiles one block takes in turn, and past what is left to one block."""
    x = np.random.default_rng(n).integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)
    want = (np.cumsum(x, dtype=np.uint64) - x).astype(np.uint32)  # 32-bit sums wrap
    with trax_lib.Context(0) as ctx:
        assert np.array_equal(ctx.prefix_sum(x), want)


@pytest.mark.parametrize("graph", [True, False])
def test_tracks_of_a_batch_without_links(trax_lib, graph):
    """One layer triplet links nothing: reading the tracks of a fresh context's batch gives none, in both modes."""
    with trax_lib.Context(0) as ctx:
        ctx.upload(events.generate(0, n_events=3))
        st = ctx.seed_batch(use_graph=graph)
        out = [np.zeros(st.n_triplets + 1, np.uint32) for _ in range(3)]
        assert st.n_triplets > 0 and st.n_links == 0 and st.n_track_entries == 0
        assert all(v.size == 0 for v in ctx.tracks(out=out)) and all(v.size == 0 for v in ctx.tracks())
