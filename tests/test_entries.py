"""The seams between the library's files and between it and Python: entries are declared in one header that their definitions see, and the
structures that Python fills have the library's sizes."""
import ctypes
import glob
import os
import re

import pytest

from beglin_b200.csrc import ops

HERE = os.path.dirname(ops.__file__)


def test_entries_are_declared_in_one_header():
    header = open(os.path.join(HERE, "entries.cuh")).read()
    declared = set(re.findall(r"\b(bg_\w+)\(", header))
    defined = {}
    for path in glob.glob(os.path.join(HERE, "*.cu")):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        assert not re.search(r'extern "C" \{|extern "C" [^;{]*;', text), f"{os.path.basename(path)} declares an entry by hand"
        for name in re.findall(r'extern "C"\s+(?:int|long long|void)\s+(bg_\w+)\(', text):
            defined[name] = path
    assert declared <= set(defined)
    assert 'include "entries.cuh"' in open(os.path.join(HERE, "common.cuh")).read()


def test_mirrored_structures_have_the_librarys_sizes(monkeypatch):
    ops.lib()                                          # (loads, and has compared them)

    class Longer(ops.LatentArgs):
        _fields_ = [("more", ctypes.c_void_p)]

    monkeypatch.setattr(ops, "_lib", None)
    monkeypatch.setattr(ops, "LatentArgs", Longer)
    with pytest.raises(ops.KernelError, match="another size"):
        ops.lib()
