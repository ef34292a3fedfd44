"""The build's inputs (CPU): every file the sources include by name decides
whether the library is up to date."""
import importlib.util
import os
import re

from conftest import ROOT

PKG = os.path.join(ROOT, "gauss-legendre-spherical-t_b200")


def test_every_included_file_is_an_input():
    spec = importlib.util.spec_from_file_location("glst_build", os.path.join(PKG, "build.py"))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    names = {os.path.basename(f) for f in build.inputs()}
    todo, seen = [f for f in os.listdir(os.path.join(PKG, "csrc")) if f.endswith((".cu", ".cpp"))], set()
    assert todo
    while todo:
        f = todo.pop()
        if f in seen:
            continue
        seen.add(f)
        assert f in names, f
        path = os.path.join(PKG, "csrc", f)
        if not os.path.exists(path):
            path = os.path.join(ROOT, "include", f)
        todo += re.findall(r'#include "([^"]+)"', open(path).read())
