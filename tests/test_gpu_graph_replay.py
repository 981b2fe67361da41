"""A session's loops stay replayable beside each other: alternating STEM, CBED and HRTEM calls each replay
their own graph."""
import numpy as np
import pytest

from totem_b200 import capi, request

pytestmark = pytest.mark.gpu


def _graph_launches(calls):
    import torch
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        calls()
    events = {e.key: e.count for e in prof.key_averages()}
    if not any(k.startswith("cuda") for k in events):
        pytest.skip("no runtime calls traced here")
    return events.get("cudaGraphLaunch", 0)


def test_alternating_calls_are_replayed(engine_lib):
    n = 64
    req = request.build_small_stem(n=n, p=n, raster=(1, 1), slices=5, mid_layer=(), focal_steps=3, sampling=0.15,
                                   begin=(0, 0))
    spec = request.hrtem_spec(n, 0.15, 200.0, 1.9525, -50.0, 1.2, 20.0, 4.0, 3)
    s = capi.Session(device=0)
    s.upload(req)

    def once():
        s.run()
        return s.download()[0], s.cbed(), s.hrtem(spec)[0]
    first = once()  # launched directly
    once()          # captured
    again = []
    assert _graph_launches(lambda: again.extend(once() for _ in range(3))) == 9
    for r in again:
        assert all(np.array_equal(a, b) for a, b in zip(first, r))
    s.close()
