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


def test_the_host_module_is_built_again_for_another_torch_and_replaced_whole(builder, monkeypatch):
    import torch
    builder.build(force=True)
    made = [cmd for cmd in builder.commands if builder.CALLS_SOURCE in cmd]
    assert len(made) == 1 and made[0][made[0].index("-o") + 1] != builder.CALLS  # written beside it, then put in its place
    assert os.listdir(os.path.dirname(builder.CALLS)).count(os.path.basename(builder.CALLS)) == 1
    assert not [n for n in os.listdir(os.path.dirname(builder.CALLS)) if n.startswith("_calls.so.")]
    with open(builder.CALLS, "ab") as f:
        f.write(builder.calls_built_for().encode())
    assert not builder.calls_need_build()
    monkeypatch.setattr(torch, "__version__", "9.9")
    assert builder.calls_need_build()


def test_a_compile_that_fails_leaves_the_host_module_as_it_is(builder, monkeypatch):
    builder.build_calls()

    def fails(cmd, **kw):
        with open(cmd[cmd.index("-o") + 1], "w") as f:
            f.write("half")
        return types.SimpleNamespace(returncode=1, stdout="", stderr="no")

    monkeypatch.setattr(builder.subprocess, "run", fails)
    with pytest.raises(RuntimeError, match="failed on cg_calls"):
        builder.build_calls()
    assert open(builder.CALLS).read() == "built" and os.listdir(os.path.dirname(builder.CALLS)).count("_calls.so") == 1
    assert not [n for n in os.listdir(os.path.dirname(builder.CALLS)) if n.startswith("_calls.so.")]
