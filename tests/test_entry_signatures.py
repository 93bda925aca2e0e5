"""The argument types of the kernel library's entry points, read from its sources, against the calls that are made."""
import ast
import ctypes
import os

import pytest

from tffinfer_b200.csrc import build
from tffinfer_b200.kernels import library


def declared():
    out = {}
    for source in build.sources():
        with open(os.path.join(build.CSRC_DIR, source), encoding="utf-8") as f:
            for name, result, types in library.function_signatures(f.read()):
                assert name not in out
                out[name] = (result, types)
    return out


def test_every_call_passes_what_the_source_declares():
    functions = declared()
    with open(library.__file__, encoding="utf-8") as f:
        tree = ast.parse(f.read())
    calls = [n for n in ast.walk(tree) if isinstance(n, ast.Call) and isinstance(n.func, ast.Attribute)
             and n.func.attr.startswith("tff_") and isinstance(n.func.value, ast.Attribute) and n.func.value.attr == "lib"]
    assert len(calls) > 50
    for call in calls:
        _, types = functions[call.func.attr]
        if not any(isinstance(a, ast.Starred) for a in call.args):
            assert len(call.args) == len(types), (call.func.attr, call.lineno)
            for arg, kind in zip(call.args, types):
                maker = arg.func.id if isinstance(arg, ast.Call) and isinstance(arg.func, ast.Name) else ""
                if maker == "_ptr":
                    assert kind is ctypes.c_void_p, (call.func.attr, call.lineno)
                elif maker == "_c_float":
                    assert kind is ctypes.c_float, (call.func.attr, call.lineno)
                elif maker == "_c_int":
                    assert kind in (ctypes.c_int, ctypes.c_longlong), (call.func.attr, call.lineno)


@pytest.mark.parametrize("params,want", [
    ("", []), ("const int* a, cudaStream_t s", [ctypes.c_void_p, ctypes.c_void_p]),
    ("long long n, float x,\n   const int k", [ctypes.c_longlong, ctypes.c_float, ctypes.c_int]),
    ("const float* const* w, // comment, with a comma\n int m", [ctypes.c_void_p, ctypes.c_int])])
def test_parameters_and_their_types(params, want):
    (name, result, types), = library.function_signatures(f"TFF_API long long tff_some_name({params}) {{ return 0; }}")
    assert name == "tff_some_name" and result is ctypes.c_longlong and types == want


def test_a_type_without_a_counterpart_is_refused():
    with pytest.raises(library.KernelError):
        library.function_signatures("TFF_API int tff_f(double x) {")


def test_arguments_are_refused_as_ctypes_refuses_them():
    """What a call passes goes through makers that take and refuse what ctypes.c_int and ctypes.c_float do."""
    import numpy as np
    import torch
    values = [3, True, -1, 2.5, 2.0, "3", None, np.int64(5), np.float64(1.5), torch.tensor(4), torch.tensor(0.5), [1], 2 ** 31]
    for maker, kind in ((library._c_int, ctypes.c_int), (library._c_float, ctypes.c_float)):
        for value in values:
            try:
                want = kind(value).value
            except TypeError:
                with pytest.raises(TypeError):
                    maker(value)
            else:
                assert kind(maker(value)).value == want, (kind, value)
    with open(library.__file__, encoding="utf-8") as f:
        assert " ll = int\n" not in f.read()
