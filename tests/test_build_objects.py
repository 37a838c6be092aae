"""Objects of an interrupted or overtaken build are not taken as current
(CPU test): nvcc's place is taken by a script that writes half an object and
fails, or during whose run a source is edited."""
import importlib.util
import os
import stat
import time

import pytest

from helpers import REPO


@pytest.fixture()
def build(tmp_path, monkeypatch):
    spec = importlib.util.spec_from_file_location("build_under_test", os.path.join(
        REPO, "planck-refactored_b200", "build.py"))
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    monkeypatch.setattr(m, "CSRC", str(tmp_path))
    monkeypatch.setattr(m, "BUILD", str(tmp_path / "o"))
    monkeypatch.setattr(m, "LIB", str(tmp_path / "lib.so"))
    monkeypatch.setattr(m, "NVCC", str(tmp_path / "nvcc"))
    monkeypatch.setattr(m, "DEPS", {"a.cu": ["a.cuh"]})
    monkeypatch.setattr(m, "_units", lambda: [("a.cu", "a.o", [])])
    for name in ("a.cu", "a.cuh"):
        (tmp_path / name).write_text("1")
        os.utime(tmp_path / name, (time.time() - 10,) * 2)

    def nvcc(body):
        (tmp_path / "nvcc").write_text(
            "#!/bin/bash\nwhile [ $# -gt 0 ]; do [ \"$1\" = -o ] && out=$2; shift; done\n" + body)
        (tmp_path / "nvcc").chmod((tmp_path / "nvcc").stat().st_mode | stat.S_IXUSR)
    m.nvcc, m.tmp = nvcc, tmp_path
    return m


def test_failed_compilation_leaves_no_object(build):
    build.nvcc("echo half > $out; exit 1\n")
    with pytest.raises(RuntimeError):
        build.build()
    assert os.listdir(build.BUILD) == [] and not os.path.exists(build.LIB)


def test_failed_link_leaves_the_old_library(build):
    (build.tmp / "lib.so").write_text("old")
    build.nvcc("case $out in *.so*) echo half > $out; exit 1;; esac; echo whole > $out\n")
    with pytest.raises(Exception):
        build.build()
    assert (build.tmp / "lib.so").read_text() == "old"
    assert sorted(p.name for p in build.tmp.iterdir() if "part" in p.name) == []


def test_source_edited_during_the_compilation(build):
    build.nvcc(f"case $out in *.so*) ;; *) sleep 0.05; echo 2 > {build.tmp}/a.cuh; sleep 0.05;; esac; echo whole > $out\n")
    build.build()
    build.nvcc(f"echo again >> {build.tmp}/calls; echo whole > $out\n")
    build.build()
    assert (build.tmp / "calls").read_text().count("again") == 2      # compiled and linked again
    build.build()
    assert (build.tmp / "calls").read_text().count("again") == 2      # nothing to do
