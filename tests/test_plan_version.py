"""CPU tests: a stored launch plan holds for the kernels it was timed on, and no
others (stratiflow_b200.autotune)."""
import json

from stratiflow_b200 import autotune as A
from tests.test_autotune import _FakeSolver

PLAN = {"xkernel": 0, "xy_bands": 3, "xslabs": 6, "z_chunks": 16, "xgroups": 16, "zkernel": 1}


def _cache(tmp_path, monkeypatch, entries):
    path = tmp_path / "plans.json"
    path.write_text(json.dumps(entries))
    monkeypatch.setenv("SF_PLAN_CACHE", str(path))
    A._memory.clear()


def test_a_plan_without_a_version_is_ignored(tmp_path, monkeypatch):
    s = _FakeSolver()
    old = f"{A.device_name(s)}|{s.N1}x{s.N2}x{s.N3}|runs {s.nrun}|step"
    _cache(tmp_path, monkeypatch, {old: PLAN})
    best, log = A.tune(s, steps=1)
    assert log                       # timed again
    assert A.load_cache()[old] == PLAN   # other versions' plans stay in the file


def test_a_plan_of_other_kernels_is_ignored(tmp_path, monkeypatch):
    s = _FakeSolver()
    monkeypatch.setattr(A, "kernels_version", lambda: "aaaa")
    _cache(tmp_path, monkeypatch, {A.plan_key(A.device_name(s), s.N1, s.N2, s.N3, s.nrun, "step"): PLAN})
    got, log = A.tune(s, steps=1)
    assert got == PLAN and not log
    monkeypatch.setattr(A, "kernels_version", lambda: "bbbb")
    _, log = A.tune(s, steps=1)
    assert log


def test_the_version_follows_the_sources(tmp_path):
    for d, text in (("a", "x"), ("b", "x"), ("c", "y")):
        (tmp_path / d).mkdir()
        (tmp_path / d / "k.cu").write_text(text)
    a, b, c = (A.kernels_version(str(tmp_path / d)) for d in "abc")
    assert a == b != c
    (tmp_path / "b" / "l.cuh").write_text("x")
    A.kernels_version.cache_clear()
    assert A.kernels_version(str(tmp_path / "b")) != a
    assert A.kernels_version() == A.kernels_version(A.CSRC)
