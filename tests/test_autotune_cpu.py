"""CPU checks of the autotuner: the cache file format and round trip, key bucketing, the choice of
the fastest candidate, and that applied values reach the library (rbw_tuning_*), with fake
timings -- no GPU needed."""
import json

import pytest

import rapidbow_b200 as rbw
from rapidbow_b200 import autotune as at


@pytest.fixture(autouse=True)
def _clean():
    at.clear()
    yield
    at.clear()


def test_bucket_and_defaults():
    assert [at.bucket(n) for n in (0, 1, 2, 3, 4, 1023, 1024, 10_000_000)] == [0, 0, 1, 1, 2, 9, 10, 23]
    for name, value in at.DEFAULTS.items():
        assert at.get_value(name, 16, 4, 10_000_000) == value


def test_choose_fastest_smallest_on_ties():
    assert at.choose({8: 3.0, 16: 2.0, 32: 2.5}) == 16
    assert at.choose({4: 1.0, 2: 1.0, 6: 1.5}) == 2


def test_tune_records_applies_and_round_trips(tmp_path):
    path = str(tmp_path / "cache.json")
    t = at.Autotuner("NVIDIA B200", 148, path)
    fake = {2: 1.9, 3: 1.2, 4: 1.1, 5: 1.3, 6: 1.4, 7: 1.5, 8: 1.6}
    calls = []

    def measure():
        v = at.get_value("assign_ctas_per_sm", 10, 0, 10_000_000)  # the value set for this trial
        calls.append(v)
        return fake[v]

    e = t.tune("assign_ctas_per_sm", 10, 0, 10_000_000, measure)
    assert calls == [2, 3, 4, 5, 6, 7, 8]
    assert e["value"] == 4 and e["bucket"] == 23 and e["default_ms"] == 1.4
    assert at.get_value("assign_ctas_per_sm", 10, 0, 9_000_000) == 4       # same bucket
    assert at.get_value("assign_ctas_per_sm", 10, 0, 1 << 24) == 6          # next bucket: default
    assert at.get_value("assign_ctas_per_sm", 10, 6, 10_000_000) == 4       # L = 0 matches any depth
    t.record("scatter_rows", 16, 4, 10_000_000, {8: 0.05, 16: 0.04, 32: 0.06})
    t.save()
    d = json.load(open(path))
    assert d["format"] == at.FORMAT and d["version"] == 1 and d["device"] == {"name": "NVIDIA B200", "sms": 148}
    assert {e["param"] for e in d["entries"]} == {"assign_ctas_per_sm", "scatter_rows"}
    at.clear()
    assert at.get_value("assign_ctas_per_sm", 10, 0, 10_000_000) == 6
    t2 = at.Autotuner("NVIDIA B200", 148, path)
    assert t2.load() and t2.apply() == 2
    assert at.get_value("assign_ctas_per_sm", 10, 0, 10_000_000) == 4
    assert at.get_value("scatter_rows", 16, 4, 10_000_000) == 16
    # a cache written for another device is not used
    assert not at.Autotuner("NVIDIA H100", 132, path).load()
    # re-recording a key replaces its entry
    t2.record("scatter_rows", 16, 4, 10_000_000, {8: 0.01, 16: 0.04, 32: 0.06})
    assert len(t2.entries) == 2 and at.get_value("scatter_rows", 16, 4, 10_000_000) == 8


def test_library_rejects_bad_values():
    with pytest.raises(rbw.RbwError) as e:
        at.set_value("scatter_rows", 16, 4, 20, 12)
    assert e.value.status == rbw.RBW_ERR_INVALID_ARG
    with pytest.raises(rbw.RbwError):
        at.set_value("assign_ctas_per_sm", 16, 0, 20, 9)
    with pytest.raises(rbw.RbwError):
        at.set_value("assign_f32_ctas_per_sm", 1, 0, 20, 2)  # branch factor out of range
    at.set_value("scatter_rows", 16, 4, 20, 32)
    assert at.get_value("scatter_rows", 16, 4, 1 << 20) == 32
    at.set_value("scatter_rows", 16, 4, 20, 0)  # 0 removes the entry
    assert at.get_value("scatter_rows", 16, 4, 1 << 20) == 16


def test_float_assign_ctas_are_what_they_say():
    """One to four CTAs per SM, each its own value: four fit and are the default, three can be asked for."""
    assert at.CANDIDATES["assign_f32_ctas_per_sm"] == (1, 2, 3, 4)
    assert at.get_value("assign_f32_ctas_per_sm", 10, 0, 1 << 20) == 4
    for v in (1, 2, 3, 4):
        at.set_value("assign_f32_ctas_per_sm", 10, 0, 20, v)
        assert at.get_value("assign_f32_ctas_per_sm", 10, 0, 1 << 20) == v
    with pytest.raises(rbw.RbwError) as e:
        at.set_value("assign_f32_ctas_per_sm", 10, 0, 20, 5)
    assert e.value.status == rbw.RBW_ERR_INVALID_ARG


class _Timed:
    """The library's timing calls over fake work: `ms` per call of what was last run."""

    def __init__(self, monkeypatch, ms):
        self.ms, self.total, self.on = ms, 0.0, False
        torch = pytest.importorskip("torch")
        monkeypatch.setattr(torch.cuda, "synchronize", lambda *a: None)
        monkeypatch.setattr(rbw, "timing_enable", lambda on: setattr(self, "on", on))
        monkeypatch.setattr(rbw, "timing_reset", lambda: setattr(self, "total", 0.0))
        monkeypatch.setattr(rbw, "timing_read", lambda name: (self.total, 1))

    def ran(self, what):
        if self.on:
            self.total += self.ms(what)


class _Voc:
    branch_factor, nb_levels = 10, 6

    def __init__(self, timed):
        self.timed, self.algos = timed, []

    def lookup(self, desc, out=None, algo="auto"):
        self.algos.append(algo)
        self.timed.ran(algo)


def test_lookup_tunables_are_timed_on_the_tensor_core_passes(monkeypatch):
    """150,000 rows of six levels go down in one launch under "auto", whatever the schedule: the candidates
    are timed by their own algorithms, and the chosen one is for the larger lookups of the same bucket."""
    import torch

    desc = torch.zeros((150_000, 128), dtype=torch.uint8)
    voc = _Voc(_Timed(monkeypatch, {"tensor_u8": 0.3, "tensor_u8_ring": 0.2}.__getitem__))
    e = at.Autotuner("x", 148, "unused").tune_lookup(voc, desc, repeats=2)
    assert set(voc.algos) == {"tensor_u8", "tensor_u8_ring"}
    assert e["value"] == 2 and e["candidates"] == {"1": 0.3, "2": 0.2}
    assert at.get_value("lookup_schedule", 10, 6, 250_000) == 2
    voc = _Voc(_Timed(monkeypatch, lambda algo: 1.0 / at.get_value("scatter_rows", 10, 6, 150_000)))
    e = at.Autotuner("x", 148, "unused").tune_lookup_regroup(voc, desc, repeats=2)
    assert set(voc.algos) == {"tensor_u8"} and e["value"] == 32


def test_builds_are_timed_once_per_grid(monkeypatch):
    """The center sums have one form and five CTAs per SM fit: no candidate is timed against itself."""
    import torch

    ctas = []
    timed = _Timed(monkeypatch, lambda c: {2: 4.0, 3: 2.0, 4: 3.0, 6: 2.5}[c])

    def build(desc, B, nb_levels, float_centers, **kw):
        ctas.append(at.get_value("assign_ctas_per_sm", B, 0, desc.shape[0]))
        timed.ran(ctas[-1])

    monkeypatch.setattr(rbw, "build_vocabulary", build)
    t = at.Autotuner("x", 148, "unused")
    e = t.tune_build(torch.zeros((5000, 128), dtype=torch.uint8), 10, 3, repeats=1)
    assert ctas == [2, 2, 3, 3, 4, 4, 6, 6]  # a warm-up and a timed build each
    assert e["value"] == 3 and e["default_ms"] == 2.5
    assert e["sums"]["value"] == at.DEFAULTS["assign_sums"] and e["sums"]["candidates"] == {"1": 2.0}
    assert {x["param"] for x in t.entries} == {"assign_sums", "assign_ctas_per_sm"}
