"""The build: what is made, from what, and what a part that cannot be made leaves of the others."""
import os
import subprocess
import sys
import types

import pytest


@pytest.fixture
def builder(monkeypatch, tmp_path):
    """The build module with its results in a folder of their own and its compilers replaced by a note of their commands."""
    from cachegen_b200 import build
    commands = []

    def run(cmd, **kw):
        commands.append(cmd)
        with open(cmd[cmd.index("-o") + 1], "w") as f:
            f.write("built")
        return types.SimpleNamespace(returncode=0, stdout="", stderr="")

    monkeypatch.setattr(build, "LIB", str(tmp_path / "lib.so"))
    monkeypatch.setattr(build, "CALLS", str(tmp_path / "_calls.so"))
    monkeypatch.setattr(build, "subprocess", types.SimpleNamespace(run=run, PIPE=subprocess.PIPE))
    csrc = build.CSRC
    monkeypatch.setattr(build, "CSRC", str(tmp_path))
    for name in build.SOURCES:
        os.symlink(os.path.join(csrc, name), tmp_path / name)
    build.commands = commands
    yield build
    del build.commands


def compiled(build):
    return sorted(os.path.basename(cmd[cmd.index("-c") + 1]) for cmd in build.commands if "-c" in cmd)


@pytest.mark.parametrize("force", [True, False])
def test_the_library_is_built_without_torch(builder, monkeypatch, capsys, force):
    monkeypatch.setitem(sys.modules, "torch", None)  # importing it raises ImportError
    assert builder.build(force=force) == builder.LIB
    assert compiled(builder) == sorted(builder.SOURCES) and os.path.exists(builder.LIB)
    assert "_calls.so was not built" in capsys.readouterr().err and not os.path.exists(builder.CALLS)


def test_the_library_is_built_without_a_host_compiler_for_the_module(builder, monkeypatch, capsys):
    def missing(cmd, **kw):
        raise FileNotFoundError(cmd[0])

    run = builder.subprocess.run
    monkeypatch.setattr(builder.subprocess, "run", lambda cmd, **kw: (run if cmd[0] == builder._nvcc() else missing)(cmd, **kw))
    assert builder.build(force=True) == builder.LIB and compiled(builder) == sorted(builder.SOURCES)
    assert "_calls.so was not built" in capsys.readouterr().err


def test_a_library_that_does_not_compile_is_an_error(builder, monkeypatch):
    monkeypatch.setattr(builder.subprocess, "run", lambda cmd, **kw: types.SimpleNamespace(returncode=1, stdout="", stderr="no"))
    with pytest.raises(RuntimeError, match="nvcc failed"):
        builder.build(force=True)
