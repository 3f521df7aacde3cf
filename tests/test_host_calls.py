"""The package's own way of calling the library (csrc/host_calls.c) passes what ctypes passes, and refuses what is no call."""
import ctypes as C
import os
import sysconfig

import pytest

from aotx_b200.library import load_library, native_call

ARGUMENTS = {"aotx_q8_matmul": (None, 0, 0, 8, 1, 32, 0, 0, 1, None, 0, 0),
             "aotx_q8_matmul_fused": (None, 0, 0, 8, 1, 32, 0, 0, 1, None, 0, 0, 0),
             "aotx_q8_dequant": (None, 0, 0, 8, 32, 0, 1, 0)}


@pytest.mark.parametrize("name", sorted(ARGUMENTS))
def test_same_answer_as_through_ctypes(name):
    lib = load_library()
    call = native_call(lib, name)
    assert call(*ARGUMENTS[name]) == getattr(lib, name)(*ARGUMENTS[name]) != 0      # no context
    for wrong in (ARGUMENTS[name][:-1], ARGUMENTS[name] + (0,), (1.5,) + ARGUMENTS[name][1:], ("x",) + ARGUMENTS[name][1:]):
        with pytest.raises(TypeError):
            call(*wrong)


@pytest.mark.parametrize("name", sorted(ARGUMENTS))
def test_none_is_a_null_pointer_and_no_number(name):
    lib = load_library()
    call = native_call(lib, name)
    good = ARGUMENTS[name]
    for i, kind in enumerate(getattr(lib, name).argtypes):
        one = good[:i] + (None,) + good[i + 1:]
        if kind is C.c_void_p:
            assert call(*one) == getattr(lib, name)(*one) != 0
            continue
        for way, error in ((call, TypeError), (getattr(lib, name), C.ArgumentError)):
            with pytest.raises(error):
                way(*one)


def test_every_argument_arrives_in_its_place():
    seen = []
    kind = C.CFUNCTYPE(C.c_int, *[C.c_void_p] * 3, C.c_uint32, C.c_uint32, C.c_uint32, C.c_void_p, C.c_int, C.c_uint32, C.c_void_p,
                       C.c_void_p, C.c_int, C.c_int)

    class Library:
        aotx_q8_matmul_fused = kind(lambda *args: seen.append(args) or 7)

    big = 0x7F1234567890
    sent = (big, big + 1, big + 2, 8, 2 ** 32 - 1, 2 ** 32 + 5, big + 3, 1, 9, None, big + 4, 2, -1)
    assert native_call(Library, "aotx_q8_matmul_fused")(*sent) == 7
    assert seen == [(big, big + 1, big + 2, 8, 2 ** 32 - 1, 5, big + 3, 1, 9, None, big + 4, 2, -1)]


def test_another_interpreter_does_not_find_the_module():
    from aotx_b200 import _host_calls, build
    build.build()
    suffix = sysconfig.get_config_var("EXT_SUFFIX")
    assert suffix != ".so" and _host_calls.__file__ == build.CALLS and build.CALLS.endswith(suffix)
    assert not os.path.exists(os.path.join(build.HERE, "_host_calls.so"))


def test_library_needs_neither_the_module_nor_python_headers(monkeypatch, tmp_path, capsys):
    import sys
    import aotx_b200
    from aotx_b200 import build
    monkeypatch.setattr(build, "CALLS", str(tmp_path / "module.so"))
    build._build_calls(str(tmp_path))
    assert "not built" in capsys.readouterr().err and not os.path.exists(build.CALLS)
    monkeypatch.delattr(aotx_b200, "_host_calls", raising=False)
    monkeypatch.setitem(sys.modules, "aotx_b200._host_calls", None)      # an import of it fails
    lib = load_library()
    for name, arguments in ARGUMENTS.items():
        assert native_call(lib, name)(*arguments) == getattr(lib, name)(*arguments) != 0
