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


def test_debug_build_checks_the_scoring_path():
    """The kernels of a batch's scoring whose indices come from tables check them in a TP3_DEBUG build."""
    for file, functions in {"kernels_lane.cu": ("lane_task", "k_couple_lane", "k_gather_lane"),
                            "kernels_hform.cu": ("k_build_H_pairs",), "kernels_tc.cu": ("k_gather_sym",),
                            "kernels_fold.cu": ("k_couple_fold",)}.items():
        with open(os.path.join(PKG, "csrc", file)) as f:
            bodies = re.split(r"^}", f.read(), flags=re.M)  # functions end at the margin
        for name in functions:
            assert any("TP3_DCHECK" in b for b in bodies if re.search(r"\b" + name + r"\([^;{]*\{", b)), name
