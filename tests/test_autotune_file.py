"""The tuner's file serves the library it was written with, and no other."""
import json
import types

import torch

from vesper_python_gb300 import _native, autotune
from vesper_python_gb300 import vesper as vg


def test_entries_of_another_library_are_not_taken(monkeypatch, tmp_path):
    path = tmp_path / "autotune.json"
    monkeypatch.setenv("VESPER_AUTOTUNE_CACHE", str(path))
    monkeypatch.setattr(autotune, "_mem", {})
    monkeypatch.setattr(vg, "search_plan", lambda *a, **k: (1, 5))
    dev = types.SimpleNamespace(device=torch.device("cpu"))
    data, mats = torch.zeros(80, 80, 80), torch.zeros(600, 3, 3)
    timed = []

    def tune():
        monkeypatch.setattr(autotune, "_mem", {})      # a new process
        del timed[:]
        return autotune.tune(dev, None, data, None, "CC", 0.0, mats)

    def search(*a, batch=0, **k):
        timed.append(batch)
        raise RuntimeError("no device")

    monkeypatch.setattr(vg, "search_device", search)
    monkeypatch.setattr(torch.cuda, "Event", lambda **k: types.SimpleNamespace(record=lambda: None))
    old = {"cpu|d=80|mode=CC": {"batch": 8, "cchunk": 1, "W": 16, "ms_per_rot": 0.01}}
    path.write_text(json.dumps(old))
    monkeypatch.setattr(autotune, "_NAMES", {dev.device: "cpu"})
    assert tune()["batch"] == 0 and timed              # written without the library's name: measured again
    entries = json.loads(path.read_text())
    (key,) = set(entries) - set(old)
    entries[key]["batch"] = 128
    path.write_text(json.dumps(entries))
    assert tune()["batch"] == 128 and not timed        # this library's entry
    monkeypatch.setattr(_native, "source_digest", lambda: "another")
    assert tune()["batch"] == 0 and timed              # another library's


def test_source_digest_is_of_the_sources():
    a = _native.source_digest()
    assert a == _native.source_digest() and len(a) == 12
