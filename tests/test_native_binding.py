"""The native call path of ``Context.op`` (primitiv_b200/binding/native.cc) without a GPU: which calls it
takes, what it hands to the ctypes path, and how a failure code comes back."""
import ctypes

import pytest

import primitiv_b200 as pb
from primitiv_b200 import capi

INVALID = 1001   # what every entry point returns for a null context


@pytest.fixture()
def calls():
    pb.lib()
    from primitiv_b200 import _native
    seen = []
    op = _native.caller(0, lambda *a: seen.append(("fallback",) + a), lambda code, name: seen.append(("fail", code, name)))
    return op, seen


@pytest.mark.parametrize("args", [(0, 5, 256, None, 4, 0.5, -1, None), (0, True, 256, 256, 2 ** 64 - 1, 1, -1, 0)])
def test_plain_arguments_reach_the_library(calls, args):
    op, seen = calls
    op("b200_unary_fw", *args)
    assert seen == [("fail", INVALID, "b200_unary_fw")]


@pytest.mark.parametrize("args", [
    ("b200_unary_fw", 0, 5, 256, ctypes.c_void_p(256), 4, 0.5, -1, None),   # a ctypes object
    ("b200_unary_fw", 0, 5, 256, 256, 4, 0.5, -1),                          # too few
    ("b200_unary_fw", 0, 5, 256, 256, None, 0.5, -1, None),                 # None for a number
    ("b200_pool_stats", 0),                                                 # not among the wrapped ones
])
def test_everything_else_goes_to_ctypes(calls, args):
    op, seen = calls
    op(*args)
    assert seen == [("fallback",) + args]


def test_wrapped_names_are_entry_points_and_errors_are_raised():
    pb.lib()
    from primitiv_b200 import _native
    op = _native.caller(0, None, capi._check)
    for name, (res, argtypes) in capi.SIGNATURES.items():
        if res is ctypes.c_int and argtypes and argtypes[0] is ctypes.c_void_p and name in ("b200_fill", "b200_gemm", "b200_matmul_fw"):
            with pytest.raises(pb.B200Error) as e:
                op(name, *[0.0 if t is ctypes.c_float else 0 for t in argtypes[1:]])
            assert e.value.code == INVALID
