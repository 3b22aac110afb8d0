"""The package build's decision of what to compile (no compiler runs: a stub writes the outputs and logs its calls)."""
import os
import stat

import pytest

from av1gpu_b200 import build as B

STUB = """#!/bin/sh
while [ $# -gt 0 ]; do
  if [ "$1" = -o ]; then echo "$2" >> "%s"; echo built > "$2"; fi
  shift
done
"""


@pytest.fixture
def tree(tmp_path, monkeypatch):
    """A package tree with the real units' names, av1core headers beside it and the stub compiler."""
    csrc, inc, log = tmp_path / "csrc", tmp_path / "ref" / "av1g", tmp_path / "log"
    csrc.mkdir()
    inc.mkdir(parents=True)
    (inc / "spec_tables.h").write_text("tables 1\n")
    (inc / "cdfctx.h").write_text("cdfs 1\n")
    for src in {u[0] for u in B.UNITS}:
        (csrc / src).write_text('#include "common.cuh"\n#include "av1g/cdfctx.h"\n')
    (csrc / "common.cuh").write_text("\n")
    for gen in ("gen_txfm.py", "txfm_gen.cuh"):
        (csrc / gen).write_text("\n")
    nvcc = tmp_path / "nvcc"
    nvcc.write_text(STUB % log)
    nvcc.chmod(nvcc.stat().st_mode | stat.S_IXUSR)
    for k, v in (("CSRC", csrc), ("LIB", tmp_path / "libisearch.so"), ("BUILD_DIR", tmp_path / "_build"), ("NVCC", nvcc),
                 ("AV1CORE_INCLUDE", inc.parent)):
        monkeypatch.setattr(B, k, str(v))

    def built():
        names = [os.path.basename(n).replace(".tmp", "") for n in log.read_text().split()] if log.exists() else []
        log.write_text("")
        return sorted(names)
    return tmp_path, built


ALL = sorted([u[1] for u in B.UNITS] + ["libisearch.so"])


def test_every_unit_follows_the_headers(tree, monkeypatch):
    """The tables come from av1core's headers: other headers, wherever they lie and whatever their dates, are compiled in."""
    tmp, built = tree
    B.build_lib()
    assert built() == ALL
    B.build_lib()
    assert built() == []
    h = tmp / "ref" / "av1g" / "cdfctx.h"
    old = h.stat().st_mtime
    h.write_text("cdfs 2\n")
    os.utime(h, (old - 1000, old - 1000))           # (a checkout's files may be older than the objects)
    B.build_lib()
    assert built() == ALL
    other = tmp / "other" / "av1g"
    other.mkdir(parents=True)
    (other / "cdfctx.h").write_text("cdfs 3\n")
    (other / "spec_tables.h").write_text("tables 1\n")
    monkeypatch.setattr(B, "AV1CORE_INCLUDE", str(other.parent))
    B.build_lib()
    assert built() == ALL
    B.build_lib()
    assert built() == []


def test_objects_of_unknown_headers_are_compiled_again(tree):
    tmp, built = tree
    (tmp / "_build").mkdir()
    for _, o, _ in B.UNITS:
        (tmp / "_build" / o).write_text("object\n")
    (tmp / "libisearch.so").write_text("library\n")
    B.build_lib()
    assert built() == ALL


def test_a_failed_compile_leaves_no_mixture(tree, monkeypatch):
    """Some units compiled from new headers, others not: the next build compiles all of them again, with old headers too."""
    tmp, built = tree
    B.build_lib()
    built()
    h = tmp / "ref" / "av1g" / "cdfctx.h"
    h.write_text("cdfs 2\n")
    good = (tmp / "nvcc").read_text()
    (tmp / "nvcc").write_text(good.replace("while", 'case "$*" in *is_k_pf*) exit 1;; esac\nwhile', 1))
    with pytest.raises(RuntimeError):
        B.build_lib(jobs=1)
    (tmp / "nvcc").write_text(good)
    h.write_text("cdfs 1\n")
    built()
    B.build_lib()
    assert built() == ALL


def test_without_headers_the_library_is_named(tree, monkeypatch, capfd):
    tmp, built = tree
    B.build_lib()
    built()
    monkeypatch.setattr(B, "AV1CORE_INCLUDE", "")
    assert B.build_lib() == B.LIB and built() == []
    assert "not compiled here" in capfd.readouterr().err
    os.remove(B.LIB)
    with pytest.raises(RuntimeError):
        B.build_lib()


def test_oracle_needs_the_reference_sources(tree, monkeypatch):
    """A checkout path without av1core in it (an empty folder) builds no oracle and is no error of the build."""
    tmp, _ = tree
    (tmp / "empty").mkdir()
    runs = []
    monkeypatch.setattr(B.subprocess, "run", lambda *a, **k: runs.append(a))
    for ref in ("", str(tmp / "empty"), str(tmp / "absent")):
        monkeypatch.setattr(B, "REF", ref)
        assert B.build_oracle() is None
    assert not runs
