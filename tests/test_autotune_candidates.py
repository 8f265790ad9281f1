"""tune() measures every kernel once (no GPU: the timing is replaced)."""
import numpy as np

from mpsim_gb300 import autotune as A


class _Lib:
    @staticmethod
    def mps_2q_workspace_bytes_mixed(*_):
        return 16


def _tune(monkeypatch, ms):
    """The entry that tune() makes of these times."""
    monkeypatch.setattr(A._native, "load", lambda: _Lib)
    monkeypatch.setattr(A, "_jobs", lambda *a: ((None,), None))
    monkeypatch.setattr(A, "_time", lambda lib, keep, S, njobs, m, n, d, cand, reps, ws: (
        ms[cand[:2]], np.ones((njobs, min(m, n)), np.float32)))
    (entry,) = A.tune([(64, 64, 64, 2)], njobs_list=(1,), device="cpu", log=lambda _: None).values()
    return entry["precision"], entry["lq_off"]


def test_noise_is_no_entry(monkeypatch):
    """A start that wins by less than the runs differ leaves the default in place."""
    ms = {("plain", 0): 1.0, ("plain", 1): 0.99, ("mixed", 0): 1.5, ("mixed", 1): 1.6}
    assert _tune(monkeypatch, ms) == ("plain", 0)
    assert _tune(monkeypatch, {**ms, ("plain", 1): 0.95}) == ("plain", 1)
    assert _tune(monkeypatch, {**ms, ("mixed", 0): 0.985}) == ("mixed", 0)
    assert _tune(monkeypatch, {**ms, ("mixed", 0): 0.96, ("mixed", 1): 0.95}) == ("mixed", 0)


def test_no_candidate_is_measured_twice(monkeypatch):
    """A block width that selects nothing is not timed beside the default, so that noise
    cannot make it an entry."""
    timed = []

    def fake_time(lib, keep, S, njobs, m, n, d, cand, reps, ws):
        timed.append(cand)
        return 1.0 - 0.01 * len(timed), np.ones((njobs, min(m, n)), np.float32)
    monkeypatch.setattr(A._native, "load", lambda: _Lib)
    monkeypatch.setattr(A, "_jobs", lambda *a: ((None,), None))
    monkeypatch.setattr(A, "_time", fake_time)
    got = A.tune([(256, 256, 256, 2)], njobs_list=(17,), device="cpu", log=lambda _: None)
    assert len({c[:2] for c in timed}) == len(timed) == 4
    (entry,) = got.values()
    assert entry["block_request"] == 0 and len(entry["ms"]) == 4
