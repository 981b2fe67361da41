"""The autotuner times the launch shapes as the engine runs them by default: its own plan of batches, not
one sequence of the largest; and bounds on a batch only where the plan comes near them."""
import types

import pytest

from totem_b200 import capi, tune


class _Session:
    """A session whose plan is ``planned`` probes a batch; every run takes a millisecond."""
    runs, planned = [], 0

    def __init__(self, device=0):
        pass

    def upload(self, req):
        pass

    def run(self, **kw):
        _Session.runs.append(kw)
        self.batch = kw["batch"] or _Session.planned

    def timing(self):
        return types.SimpleNamespace(slice_loop_ms=1.0, batch=self.batch)

    def close(self):
        pass


@pytest.mark.parametrize("planned,bounds", [(18, False), (2048, True)])  # 36 MiB and 4 GiB of 512^2 waves
def test_tuner_times_the_engines_own_plan(monkeypatch, planned, bounds):
    monkeypatch.setattr(capi, "Session", _Session)
    monkeypatch.setattr(tune, "workload", lambda n: types.SimpleNamespace(height=n, probe_slices=1000, depth=4096, slices=20,
                                                                         p_height=1024))
    _Session.runs, _Session.planned = [], planned
    entry = tune.tune_size(512, log=lambda m: None)
    timed = [r for r in _Session.runs if r.get("skip_transmission")]
    assert timed[0]["batch"] == 0
    assert {r["batch"] for r in timed} == ({0, 512, 1024} if bounds else {0})
    assert entry["batch_mib"] in tune.BATCH_MIB
