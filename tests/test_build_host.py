"""The build's staleness check covers every file the units include."""
import importlib.util
import re
from pathlib import Path

PKG = Path(__file__).resolve().parent.parent / "volumefluxes.jl_gb300"


def test_every_included_file_is_a_source():
    spec = importlib.util.spec_from_file_location("build_native", PKG / "build_native.py")
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    todo, seen = [build.CSRC / unit for unit in build.UNITS], set()
    while todo:
        f = todo.pop()
        if f in seen:
            continue
        seen.add(f)
        for name in re.findall(r'^#include "(.+)"', f.read_text(), re.M):
            todo += [p.resolve() for p in (f.parent / name, build.INCLUDE / name) if p.exists()]
    assert len(seen) > len(build.UNITS)
    assert seen <= set(build.sources()), seen - set(build.sources())
