"""Launch structure of the chain: time marks."""
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
