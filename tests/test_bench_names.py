"""Every global name the bench's functions read exists: the sections that need
a GPU, and with it the printed line, cannot fail on a name here unseen."""

import builtins
import dis
import os
import sys
import types

from conftest import ROOT

sys.path.insert(0, ROOT)

import bench  # noqa: E402


def _globals_read(code):
    names = {i.argval for i in dis.get_instructions(code)
             if i.opname in ("LOAD_GLOBAL", "LOAD_NAME")}
    for const in code.co_consts:
        if isinstance(const, types.CodeType):
            names |= _globals_read(const)
    return names


def test_functions_read_only_names_that_exist():
    missing = {}
    for name, f in vars(bench).items():
        bodies = [f] if isinstance(f, types.FunctionType) else [
            m for m in vars(f).values() if isinstance(m, types.FunctionType)
        ] if isinstance(f, type) else []
        for body in bodies:
            if body.__module__ != "bench":
                continue
            lost = {n for n in _globals_read(body.__code__)
                    if not hasattr(bench, n) and not hasattr(builtins, n)}
            if lost:
                missing[f"{name}.{body.__name__}"] = sorted(lost)
    assert not missing, missing
