"""The autotuner times each distinct form of a batch once: the geometric reconstruction has no row
tiles, so candidates that differ in them alone are one and the same pass and share a time."""
import types

import numpy as np

import viss_recon_shade_gb300 as V
from viss_recon_shade_gb300 import api


class _Event:
    clock = 0.0

    def __init__(self, enable_timing=False):
        pass

    def record(self):
        self.t = _Event.clock

    def synchronize(self):
        pass

    def elapsed_time(self, other):
        return other.t - self.t


class _Batch:
    def __init__(self, cfg):
        self.cfg, self.J, self.row_off = cfg, 100, np.array([0, 10])
        self.u = types.SimpleNamespace(device="cuda:0")
        self.timed = []

    def set_tuning(self, t):
        self.t = t

    def step(self):
        self.timed.append(self.t)
        _Event.clock += 1.0 + 0.01 * len(self.timed)


def _run(monkeypatch, cfg):
    monkeypatch.setattr(api.torch.cuda, "get_device_name", lambda d=None: "test")
    monkeypatch.setattr(api.torch.cuda, "Event", _Event)
    b = _Batch(cfg)
    best = V.autotune(b, use_cache=False)
    report = V.autotune_report(b)
    assert [t for t, _ in report] == V.tuning_candidates() and b.t == best
    assert best == report[int(np.argmin([ms for _, ms in report]))][0]
    return b, dict((id(t), ms) for t, ms in report), report


def test_geometric_candidates_are_timed_once(monkeypatch):
    b, _, report = _run(monkeypatch, V.DftConfig.geometric())
    keys = [(t.tile & 1, t.rec_items, t.ctas_per_sm, t.vis_split) for t in b.timed]
    assert len(keys) == 2 * len(set(keys))  # a warm-up and a timed run of each
    assert set(keys) == {(t.tile & 1, t.rec_items, t.ctas_per_sm, t.vis_split) for t in V.tuning_candidates()}
    ms = {}
    for t, x in report:
        assert ms.setdefault((t.tile & 1, t.rec_items, t.ctas_per_sm, t.vis_split), x) == x


def test_other_masks_time_every_candidate(monkeypatch):
    b, _, _ = _run(monkeypatch, V.DftConfig())
    assert len(b.timed) == 2 * len(V.tuning_candidates())
