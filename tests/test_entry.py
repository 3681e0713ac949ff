"""build() where the reference's sources are absent (CPU)."""
import importlib

import pytest


@pytest.mark.parametrize("sources", ["none", "empty", "there"])
def test_the_reference_is_built_only_from_its_sources(monkeypatch, tmp_path, sources):
    ref = tmp_path / "reference"
    if sources != "none":
        ref.mkdir()
    if sources == "there":
        (ref / "accel").mkdir()
    monkeypatch.setenv("PSY_REFERENCE_DIR", str(ref))
    entry = importlib.reload(importlib.import_module("__graft_entry__"))
    from psychopath_cpp_b200 import build as b
    targets = []
    monkeypatch.setattr(b, "build", lambda: None)
    monkeypatch.setattr(entry.subprocess, "run", lambda cmd, **kw: targets.append(cmd[3]))
    entry.build()
    assert targets == (["port", "ref"] if sources == "there" else ["port"])
    monkeypatch.undo()
    importlib.reload(entry)
