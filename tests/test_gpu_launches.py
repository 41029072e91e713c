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
