"""When the extension module of the native call path is compiled again: it calls the C ABI through addresses and reads torch's tensors at
the offsets of the headers it saw, so a module older than either would pass arguments in the wrong places (nothing is compiled here)."""
import importlib.util
import os
import re

import pytest

PACKAGE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fp6_marlin_b200")


@pytest.fixture
def builder(tmp_path, monkeypatch):
    """build.py with copies of the sources, a torch of two files and a compiler that only writes its output."""
    spec = importlib.util.spec_from_file_location("_build_under_test", os.path.join(PACKAGE, "build.py"))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    root = tmp_path / "repo"
    for name in ("fp6_marlin_b200/csrc/py_call.cpp", "include/fp6m.h"):
        (root / name).parent.mkdir(parents=True, exist_ok=True)
        (root / name).write_text(open(os.path.join(os.path.dirname(PACKAGE), name)).read())
    torch_dir = tmp_path / "torch"
    torch_dir.mkdir()
    (torch_dir / "version.py").write_text("__version__ = '1.0'\n")
    monkeypatch.setattr(importlib.util, "find_spec", lambda name: type("Spec", (), {"submodule_search_locations": [str(torch_dir)]}))
    for name, value in vars(build).items():         # every path below the repository, whatever its name
        old = os.path.dirname(PACKAGE)
        if isinstance(value, str) and value.startswith(old):
            monkeypatch.setattr(build, name, str(root) + value[len(old):])
        elif isinstance(value, list) and any(str(v).startswith(old) for v in value):
            monkeypatch.setattr(build, name, [str(root) + v[len(old):] if v.startswith(old) else v for v in value])
    compiled = []

    def compiler(command, check):
        compiled.append(command)
        open(command[command.index("-o") + 1], "w").close()

    monkeypatch.setattr(build.subprocess, "run", compiler)
    build.root, build.torch_dir, build.compiled = root, torch_dir, compiled
    return build


def _age(path):
    """A file that changed long ago: its time stamp alone does not show the change."""
    os.utime(path, (1, 1))


def _builds(build):
    before = len(build.compiled)
    build.build_call()
    return len(build.compiled) - before


def test_an_unchanged_tree_is_not_compiled_again(builder):
    assert [_builds(builder) for _ in range(3)] == [1, 0, 0]
    os.remove(builder.CALL_PATH)
    assert _builds(builder) == 1


@pytest.mark.parametrize("what", ["fp6_marlin_b200/csrc/py_call.cpp", "include/fp6m.h", "torch"])
def test_a_change_is_compiled(builder, what):
    path = builder.torch_dir / "version.py" if what == "torch" else builder.root / what
    _builds(builder)
    path.write_text(path.read_text() + ("__version__ = '2.0'\n" if what == "torch" else "/* changed */\n"))
    _age(path)
    assert _builds(builder) == 1
    assert _builds(builder) == 0


def test_the_module_has_the_types_of_the_c_abi():
    """No restated signature that could differ from the declaration."""
    source = open(os.path.join(PACKAGE, "csrc", "py_call.cpp")).read()
    assert '#include "../../include/fp6m.h"' in source
    for name in ("fp6m_mul", "fp6m_mul_fused", "fp6m_mul_scratch_bytes"):
        assert f"decltype(&{name})" in source
    assert not re.search(r"typedef\s", source)
