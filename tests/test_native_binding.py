"""The native call path of ``Context.op`` (primitiv_b200/binding/native.cc) without a GPU: which calls it
takes, what it hands to the ctypes path, and how a failure code comes back."""
import ctypes
import gc
import subprocess
import sys
import sysconfig
import weakref

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


@pytest.fixture()
def destroyed(monkeypatch):
    """Contexts without a GPU: creation hands out an address that nothing follows, destruction notes it."""
    real, gone = pb.lib(), []

    class Library:
        def b200_ctx_create(self, device, out):
            out._obj.value = 4096
            return 0

        def b200_ctx_destroy(self, h):
            gone.append(h.value)

        def __getattr__(self, name):
            return getattr(real, name)

    stand_in = Library()
    monkeypatch.setattr(capi, "lib", lambda: stand_in)
    yield gone
    gc.collect()


FILL = ("b200_fill", 0, 256, 4, 0.5, None)


def test_a_kept_op_keeps_its_context_alive(destroyed):
    c = pb.Context(0)
    op, alive = c.op, weakref.ref(c)
    del c
    gc.collect()
    assert alive() is not None and not destroyed
    del op
    assert alive() is None and destroyed == [4096]   # at once: no cycle holds a context until the next collection


def test_a_closed_context_has_a_null_pointer(destroyed):
    c = pb.Context(0)
    op = c.op
    c.close()
    c.close()
    assert destroyed == [4096]
    for call in (op, c.op):
        with pytest.raises(pb.B200Error) as e:
            call(*FILL)
        assert e.value.code == INVALID


def test_a_subclass_can_put_its_own_op_in_place(destroyed):
    class Other(pb.Context):
        def op(self, name, *args):
            raise AssertionError("looked up, not called")

    assert Other(0).op.__func__ is Other.op


def test_an_object_without_an_address_goes_to_the_fallback():
    pb.lib()
    from primitiv_b200 import _native
    seen = []

    class Other:
        op = _native.caller(None, lambda *a: seen.append(a), None)

    o = Other()
    o.op(*FILL)
    for address in (None, "0", 2 ** 70):
        o._address = address
        o.op(*FILL)
    assert seen == [(o,) + FILL] * 4


def test_the_native_form_is_this_interpreters_own():
    pb.lib()
    from primitiv_b200 import _native
    assert _native.__file__.endswith(sysconfig.get_config_var("EXT_SUFFIX"))


def test_calls_go_without_the_native_form():
    """Where there is none (no Python headers, another interpreter) every call goes through ctypes."""
    code = """if True:
        import sys
        sys.modules["primitiv_b200._native"] = None     # what an import of it then finds
        import primitiv_b200 as pb
        pb.lib()
        c = pb.Context.__new__(pb.Context)
        c._h = None
        try:
            c.matmul_fw(0, 256, 256, 256, 1, 1, 1, 1, 1)
        except pb.B200Error as e:
            print(e.code)
    """
    r = subprocess.run([sys.executable, "-c", code], cwd=capi._PKG + "/..", capture_output=True, text=True)
    assert r.stdout.split() == [str(INVALID)], r.stdout + r.stderr
