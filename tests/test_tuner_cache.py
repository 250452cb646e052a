"""The tuner's cache: entries of an earlier version, timed on other kernels, are
not used."""
import json

from conftest import load_package

pkg = load_package()
from special_topics_b200 import autotune as T  # noqa: E402


def test_entries_of_an_earlier_version_are_not_used(tmp_path, monkeypatch):
    path = tmp_path / "tiling.json"
    monkeypatch.setattr(T, "CACHE", str(path))
    path.write_text(json.dumps({"f32-table:8x8x8": {"chunk": 8, "rows": 4, "streams": 4}}))
    assert T._load() == {}
    T._store({"f32-table:8x8x8": {"chunk": 2, "rows": 2}})
    assert T._load() == {"f32-table:8x8x8": {"chunk": 2, "rows": 2}}
    for broken in ("", "[]", "3", '{"version": 2}'):
        path.write_text(broken)
        assert T._load() == {}
