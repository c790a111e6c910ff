"""CPU suite: the binding of asp_spmv without ctypes (csrc/python/call.c) refuses and accepts what the ctypes one did."""
import ctypes as C
import importlib.machinery
import os
import sys
import sysconfig

import pytest

import alphasparse_b200
from alphasparse_b200 import capi


def bound():
    handle, plans = C.c_void_p(), (C.c_void_p * 1)()
    call = capi._native().Spmv(C.cast(capi.lib().asp_spmv, C.c_void_p).value, C.addressof(handle), C.addressof(plans), 1)
    return call, handle, plans


@pytest.mark.parametrize("args", [(None, 1, 2), (1, None, 2), (1.0, 2, 2), (1, 2), (1, 2, 2, 2), (1, 2, "auto")])
def test_only_ints_are_taken(args):
    call, *keep = bound()
    with pytest.raises(TypeError):
        call(*args)
    with pytest.raises(TypeError):
        call(1, 2, zero_y=2)


@pytest.mark.parametrize("x,y", [(0, 0), (1, 0), (0, 1), (2**64 - 16, 2**63), (-16, 1 << 70)])
def test_handles_are_read_at_the_call(x, y):
    """A context that is closed is NULL to the library, whatever the pointers are (taken modulo 2^64, as ctypes takes them)."""
    call, handle, plans = bound()
    assert call(x, y, 2) == 1 and b"NULL" in capi.lib().asp_last_error()


def test_a_call_without_plan_or_with_other_pointers_falls_back():
    group = object.__new__(capi.PlanGroup)
    group.n, group._plans = 1, (C.c_void_p * 1)()
    group.ctx = object.__new__(capi.Context)
    group.ctx._h = C.c_void_p()
    group._call = capi._native().Spmv(C.cast(capi.lib().asp_spmv, C.c_void_p).value, C.addressof(group.ctx._h), C.addressof(group._plans), 1)
    for x in (16, None, C.c_void_p(16)):
        with pytest.raises(capi.AspError):
            group.spmv(x, 16)
    with pytest.raises(C.ArgumentError):
        group.spmv(1.5, 16)


def test_calls_without_the_binding_go_through_ctypes(monkeypatch):
    """Where only the library has been built, the same calls are taken and refused."""
    monkeypatch.setitem(sys.modules, "alphasparse_b200._call", None)  # (as if there were no such file)
    monkeypatch.delattr(alphasparse_b200, "_call", raising=False)
    group = object.__new__(capi.PlanGroup)
    group.n, group._plans = 1, (C.c_void_p * 1)()
    group.ctx = object.__new__(capi.Context)
    group.ctx._h = C.c_void_p()
    group._call = capi._bind_spmv(group.ctx._h, group._plans, 1)
    assert group._call(16, 32, 2) == 1 and b"NULL" in capi.lib().asp_last_error()
    for x in (16, None, C.c_void_p(16)):
        with pytest.raises(capi.AspError):
            group.spmv(x, 16)
    with pytest.raises(C.ArgumentError):
        group.spmv(1.5, 16)


def test_the_binding_is_for_this_python_alone():
    """It uses more of Python's interface than other versions share: they must not find it."""
    suffix = sysconfig.get_config_var("EXT_SUFFIX")
    assert suffix != ".so" and suffix in importlib.machinery.EXTENSION_SUFFIXES
    assert capi._native().__file__.endswith("_call" + suffix)
    assert not os.path.exists(os.path.join(os.path.dirname(capi.__file__), "_call.so"))


def test_the_build_does_without_headers_or_compiler(monkeypatch, tmp_path):
    import __graft_entry__ as entry

    monkeypatch.delenv("CC", raising=False)
    monkeypatch.setattr(entry, "_call_path", lambda: str(tmp_path / "_call.so"))
    assert "Python.h" in entry._build_call(include=str(tmp_path))
    assert "compiler" in entry._build_call(compilers=("no-such-compiler",))
    assert not os.listdir(tmp_path)
    assert entry._build_call() is None and os.listdir(tmp_path) == ["_call.so"]
