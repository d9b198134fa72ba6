"""When the in-tree libraries count as out of date: a source or the header is younger than one of them, or _native.so was compiled for another
Python or torch.  Not when an object file is: the build writes those beside the sources, some of them after _native.so."""
import os

import pytest

from kiln_b200 import build


@pytest.fixture
def tree(tmp_path, monkeypatch):
    csrc = tmp_path / "pkg" / "csrc"
    csrc.mkdir(parents=True)
    (tmp_path / "include").mkdir()
    files = {"cu": csrc / "a.cu", "h": csrc / "b.h", "o": csrc / "a.o", "header": tmp_path / "include" / "kiln_w4a16.h",
             "lib": tmp_path / "pkg" / "lib.so", "native": tmp_path / "pkg" / "_native.so"}
    for i, f in enumerate(files.values()):
        f.write_bytes(b"\0" + build._native_key().encode() + b"\0")
        os.utime(f, (1000, 1000))
    for name, value in [("HERE", tmp_path / "pkg"), ("CSRC", csrc), ("LIB", files["lib"]), ("NATIVE", files["native"])]:
        monkeypatch.setattr(build, name, str(value))
    os.utime(files["lib"], (2000, 2000))
    os.utime(files["native"], (1990, 1990))
    return files


@pytest.mark.parametrize("touched,stale", [("o", False), ("cu", True), ("h", True), ("header", True)])
def test_sources_decide(tree, touched, stale):
    assert not build._stale()
    os.utime(tree[touched], (1995, 1995))
    assert build._stale() == stale


def test_another_torch_decides(tree):
    tree["native"].write_bytes(build._native_key().replace("torch ", "torch 1").encode())
    os.utime(tree["native"], (1990, 1990))
    assert build._stale()


def test_the_installed_one_is_up_to_date():
    assert build._built_for_this_torch()
