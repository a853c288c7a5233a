"""The native calls of the library's entry points take, refuse and return what ctypes does: every signature, with a Python function as the entry point."""

import ctypes
import importlib.machinery
import importlib.util

import pytest

from miniserve_b200.kernels import build

KINDS = {"pointer": ctypes.c_void_p, "int": ctypes.c_int, "float": ctypes.c_float, "longlong": ctypes.c_longlong}
VALUES = {"pointer": [None, 0, 140737488355327, 2 ** 64 - 1, -1, True], "int": [0, -1, 2 ** 31 - 1, -2 ** 31, 2 ** 32 + 5, 2 ** 70 + 3, False],
          "float": [0.0, 0.1, -1.5, float("inf"), 3, True], "longlong": [0, -1, 2 ** 63 - 1, -2 ** 63, 2 ** 64 + 9, True]}


@pytest.fixture(scope="module")
def module():
    path = build.calls_path()
    if path is None:
        pytest.skip("no compiler or headers of the interpreter")
    loader = importlib.machinery.ExtensionFileLoader(build.CALLS_NAME, str(path))
    loaded = importlib.util.module_from_spec(importlib.util.spec_from_loader(build.CALLS_NAME, loader))
    loader.exec_module(loaded)
    return loaded


def outcome(function, arguments, seen):
    del seen[:]
    try:
        return "result", function(*arguments), list(seen)
    except Exception as error:
        return type(error), str(error)


@pytest.mark.parametrize("name", sorted(n for n, (result, _) in build.exported_signatures().items() if result in ("int", "longlong")))
def test_as_ctypes(module, name):
    result, kinds = build.exported_signatures()[name]
    seen = []

    def function(*arguments):
        seen.extend(arguments)
        return -3

    general = ctypes.CFUNCTYPE(KINDS[result], *(KINDS[k] for k in kinds))(function)
    # (the general one is only for what the trampoline does not take: another function here, that says it was called)
    entry = module.entry(name, ctypes.cast(general, ctypes.c_void_p).value, general)
    for turn in range(7):
        arguments = [VALUES[k][(turn + i) % len(VALUES[k])] for i, k in enumerate(kinds)]
        assert outcome(entry, arguments, seen) == outcome(general, arguments, seen)
    usual = [VALUES[k][1] for k in kinds]
    direct = module.entry(name, ctypes.cast(general, ctypes.c_void_p).value, lambda *arguments: "general")
    assert direct(*usual) == -3
    for wrong in [usual[:-1], usual + [1], ["x"] + usual[1:], usual[:-1] + [ctypes.c_void_p(8)], usual[:-1] + [1.5]]:
        if kinds and not (kinds[-1] == "float" and wrong[-1:] == [1.5] and len(wrong) == len(kinds)):
            assert direct(*wrong) == "general"
    entry.restype = ctypes.c_int
    assert entry.restype is ctypes.c_int


@pytest.fixture
def elsewhere(tmp_path, monkeypatch):
    """A build folder of its own."""
    monkeypatch.setattr(build, "_build_dir", lambda: tmp_path)
    return tmp_path


def test_a_module_that_does_not_load_leaves_the_calls_to_ctypes(module, elsewhere, monkeypatch):
    from miniserve_b200 import kernels

    broken = elsewhere / "broken.so"
    broken.write_bytes(b"not a module")
    monkeypatch.setattr(build, "calls_path", lambda: broken)

    class Library:
        def __getattr__(self, name):
            raise AssertionError("nothing is replaced")

    kernels._take_calls(Library())


def test_another_interpreters_module_stays(module, elsewhere):
    ours = elsewhere / f"{build.CALLS_NAME}_{build.sysconfig.get_config_var('SOABI')}_0123456789abcdef.so"
    theirs = elsewhere / f"{build.CALLS_NAME}_cpython-399-x86_64-linux-gnu_0123456789abcdef.so"
    for path in (ours, theirs):
        path.write_bytes(b"")
    built = build.calls_path()
    assert built.is_file() and theirs.is_file() and not ours.is_file()


def test_a_compiler_that_refuses_is_asked_once(module, elsewhere, monkeypatch):
    asked = []

    class Refusal:
        returncode, stderr = 1, "no"

    monkeypatch.setattr(build.subprocess, "run", lambda command, **_: asked.append(command) or Refusal())
    assert build.calls_path() is None and build.calls_path() is None and len(asked) == 1
    assert [path.suffix for path in elsewhere.iterdir()] == [".refused"]
