"""The build's dependencies: a change of any file that a translation unit includes rebuilds the library."""
import importlib.util
import os
import re

PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "threephotons.jl_gb300")


def test_every_included_file_is_a_dependency():
    spec = importlib.util.spec_from_file_location("tp3_build", os.path.join(PKG, "build.py"))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    deps = {os.path.realpath(d) for d in build._deps()}
    todo, seen = list(build.sources()), set()
    while todo:
        path = os.path.realpath(todo.pop())
        if path in seen:
            continue
        seen.add(path)
        with open(path) as f:
            todo += [os.path.join(os.path.dirname(path), i) for i in re.findall(r'#include "([^"]+)"', f.read())]
    assert seen <= deps, sorted(seen - deps)
