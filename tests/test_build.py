"""What a built file was built from decides whether it is built again (gpt.c_b200/build.py); no compiler runs here."""
import importlib.metadata
import os
import shutil
import types

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture
def tree(tmp_path, monkeypatch):
    """A copy of the sources with its own build module, whose compilers write an empty file and are counted."""
    from __graft_entry__ import _load_file

    for d in ("gpt.c_b200/csrc", "include"):
        shutil.copytree(os.path.join(HERE, "..", d), tmp_path / d)
    shutil.copy(os.path.join(HERE, "..", "gpt.c_b200", "build.py"), tmp_path / "gpt.c_b200" / "build.py")
    build = _load_file("build_under_test", str(tmp_path / "gpt.c_b200" / "build.py"))
    built = []

    def compiler(cmd, **_):
        out = cmd[cmd.index("-o") + 1]
        open(out, "w").close()
        built.append(os.path.basename(out))
        return types.SimpleNamespace(returncode=0, stdout="", stderr="")

    monkeypatch.setattr(build.subprocess, "run", compiler)

    def run():
        built.clear()
        build.build()
        return sorted(built)

    assert run() == ["gptc_b200_calls.so", "libattn_sm100.so"] and run() == []
    return types.SimpleNamespace(path=tmp_path, build=build, run=run)


BOTH = ["gptc_b200_calls.so", "libattn_sm100.so"]


@pytest.mark.parametrize("name", sorted(os.listdir(os.path.join(HERE, "..", "include"))))
def test_every_public_header_counts_for_both(tree, name):
    with open(tree.path / "include" / name, "a") as f:
        f.write("/* */")
    os.utime(tree.path / "include" / name, (1, 1))  # older than what was built, as after a checkout
    assert tree.run() == BOTH and tree.run() == []


@pytest.mark.parametrize("name,expect", [("tc05.cuh", BOTH), ("xent_sm100.cu", ["libattn_sm100.so"]),
                                         ("torch_calls.cpp", ["gptc_b200_calls.so"])])
def test_sources_count_for_what_they_are_in(tree, name, expect):
    with open(tree.path / "gpt.c_b200" / "csrc" / name, "a") as f:
        f.write("// ")
    assert set(expect) <= set(tree.run()) and tree.run() == []


def test_another_torch_rebuilds_the_extension(tree, monkeypatch):
    monkeypatch.setattr(importlib.metadata, "version", lambda name: "0.0")
    assert tree.run() == ["gptc_b200_calls.so"] and tree.run() == []


def test_a_missing_file_or_stamp_is_built(tree):
    os.remove(tree.build.LIB)
    assert "libattn_sm100.so" in tree.run()
    os.remove(tree.build.CALLS + ".stamp")
    assert tree.run() == ["gptc_b200_calls.so"]
