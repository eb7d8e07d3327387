"""When the host path's object is compiled again."""

import os

import pytest


@pytest.fixture
def obj(tmp_path):
    from sageattention_b200 import build
    path = str(tmp_path / "native.o")
    for p, text in ((path, ""), (path + ".tag", build._native_tag(["c++", "-O2"]))):
        with open(p, "w") as f:
            f.write(text)
    return path


def test_object_of_this_torch_is_kept(obj):
    from sageattention_b200 import build
    assert not build._native_stale(obj, ["c++", "-O2"])


def test_object_of_another_torch_is_stale(obj, monkeypatch):
    import torch
    from sageattention_b200 import build
    monkeypatch.setattr(torch, "__version__", "99.0")
    assert build._native_stale(obj, ["c++", "-O2"])


def test_other_command_older_object_or_no_stamp_is_stale(obj):
    from sageattention_b200 import build
    assert build._native_stale(obj, ["c++", "-O3"])
    os.utime(obj, (1, 1))
    assert build._native_stale(obj, ["c++", "-O2"])
    os.utime(obj)
    os.remove(obj + ".tag")
    assert build._native_stale(obj, ["c++", "-O2"])
