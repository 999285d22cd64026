"""What build.build() makes, with a compiler that only writes the file it is asked for."""
import os
import sys
import pytest
from gaac_b200 import build


@pytest.fixture
def fake(tmp_path, monkeypatch):
    """The library and the module under tmp_path, by the compilers `cc` and `c++` there; made(name): their command lines."""
    log = tmp_path / "log"
    for name in ("cc", "c++"):
        tool = tmp_path / name
        tool.write_text(f'#!/bin/sh\necho {name} "$@" >> {log}\nwhile [ $# -gt 0 ]; do if [ "$1" = -o ]; then echo "$FAKE_OUTPUT" > "$2"; fi; shift; done\n')
        tool.chmod(0o755)
    monkeypatch.setenv("NVCC", str(tmp_path / "cc")); monkeypatch.setenv("CXX", str(tmp_path / "c++"))
    monkeypatch.setattr(build, "LIB", str(tmp_path / "lib.so")); monkeypatch.setattr(build, "HOST", str(tmp_path / "_host.so"))
    monkeypatch.setattr(build, "SOURCES", ["gaac_noalloc.cu"])
    monkeypatch.setenv("FAKE_OUTPUT", "what " + build._built_for().decode() + " needs")
    monkeypatch.setattr(build.os.path, "join", lambda *a, join=os.path.join: join(str(tmp_path), *a[1:]) if a[0] == "/tmp" else join(*a))

    def made(name):
        lines = log.read_text().splitlines() if log.exists() else []
        return sum(line.startswith(name + " ") for line in lines)
    return made


def test_the_library_and_the_module(fake):
    assert build.build() == build.LIB and os.path.exists(build.LIB) and os.path.exists(build.HOST)
    assert fake("cc") == 2 and fake("c++") == 1
    os.remove(build.HOST)
    build.build()                                     # only what is missing
    assert fake("cc") == 2 and fake("c++") == 2


@pytest.mark.parametrize("missing", ["torch", "compiler"])
def test_the_library_alone(fake, monkeypatch, missing):
    if missing == "torch": monkeypatch.setitem(sys.modules, "torch", None)
    else: monkeypatch.setenv("CXX", "/nonexistent/c++")
    assert build.build() == build.LIB and os.path.exists(build.LIB) and not os.path.exists(build.HOST)
    assert fake("cc") == 2


@pytest.mark.parametrize("found", ["ABI 3, torch %s", "ABI 4, torch 1.0", ""])
def test_a_module_for_another_abi_or_torch_is_built_again(fake, monkeypatch, found):
    import torch
    build.build()
    build.build()
    assert fake("c++") == 1
    with open(build.HOST, "w") as f: f.write(found % torch.__version__ if "%s" in found else found)
    build.build()
    assert fake("cc") == 2 and fake("c++") == 2


def test_a_module_of_another_interpreter_is_not_found():
    import importlib.machinery
    import sysconfig
    assert build.HOST.endswith(sysconfig.get_config_var("EXT_SUFFIX")) and sysconfig.get_config_var("EXT_SUFFIX") in importlib.machinery.EXTENSION_SUFFIXES


@pytest.mark.parametrize("built_for", ["ABI 3, torch %s", "ABI 4, torch 1.0", None])
def test_a_module_for_another_abi_or_torch_is_not_called(monkeypatch, built_for):
    import types
    import torch
    import gaac_b200
    from gaac_b200 import _lib
    module = types.SimpleNamespace(bind=lambda handle: pytest.fail("bound"), __file__="_host.so")
    if built_for: module.built_for = built_for % torch.__version__ if "%s" in built_for else built_for
    _lib.host()
    monkeypatch.setattr(gaac_b200, "_host", module); monkeypatch.setattr(_lib, "_host", None)
    with pytest.raises(RuntimeError, match="was built for"): _lib.host()
