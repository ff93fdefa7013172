"""Cached tuning choices belong to the build that they were timed on."""
from types import SimpleNamespace

from gde import _build, tune


def test_another_build_has_another_key(tmp_path, monkeypatch):
    graph = SimpleNamespace(n=10, cap=20, vol=20.0)
    monkeypatch.setattr(_build, "BUILD", str(tmp_path))
    monkeypatch.setattr(_build, "LIB", str(tmp_path / "libgde.so"))

    def key(stamp=None, lib=None):
        for name, text in (("libgde.stamp", stamp), ("libgde.so", lib)):
            (tmp_path / name).unlink(missing_ok=True)
            if text is not None:
                (tmp_path / name).write_text(text)
        return tune._graph_key(graph, 0, "fp32", 64, None)

    keys = [key(stamp="a"), key(stamp="b"), key(lib="a"), key(lib="b")]
    assert len(set(keys)) == 4 and key(stamp="a") == keys[0]
