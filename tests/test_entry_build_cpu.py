"""build() needs the reference's sources for the pinned oracle only: an absent or empty
reference tree leaves that part out and the rest is built."""

import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_build_without_the_reference_sources(tmp_path, monkeypatch):
    sys.path.insert(0, ROOT)
    import __graft_entry__ as entry

    commands = []
    monkeypatch.setattr(entry.subprocess, "run", lambda command, **kwargs: commands.append(command))
    monkeypatch.setattr(entry, "REFERENCE", str(tmp_path))  # exists and is empty
    monkeypatch.setitem(sys.modules, "build", type(sys)("build"))
    sys.modules["build"].build = lambda: None
    entry.build()
    assert [c[4] for c in commands if c[0] == "make"] == ["all"]
