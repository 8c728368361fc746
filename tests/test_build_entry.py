"""build() without the reference's sources: an empty folder in their place is no tree."""
import __graft_entry__ as entry
from multislice_gb300 import build as lib


def test_build_skips_the_reference_objects_without_their_sources(tmp_path, monkeypatch):
    runs = []
    monkeypatch.setattr(lib, "build", lambda: None)
    monkeypatch.setattr(entry.subprocess, "run", lambda *a, **k: runs.append(a))
    monkeypatch.setattr(entry, "REFERENCE", str(tmp_path))
    entry.build()
    assert not runs
    (tmp_path / "ImageSimulation").mkdir()
    entry.build()
    assert len(runs) == 1
