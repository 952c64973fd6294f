"""CPU: the extension module of the launch path is used with the interpreter and the torch it was made for, and a tree without a usable one says so."""
import os
import subprocess
import sys
import sysconfig

import pytest

from conftest import ROOT


def imported_with(setup):
    """(whether the native path is on, the warnings) of an import of ops behind `setup`."""
    code = ("import sys, types, warnings\n" + setup + "\nwith warnings.catch_warnings(record=True) as w:\n    warnings.simplefilter('always')\n    from fovi_b200 import ops\n"
            "print(ops._native is not None, [str(x.message) for x in w if 'launch path' in str(x.message)])")
    out = subprocess.run([sys.executable, "-c", code], check=True, cwd=ROOT, capture_output=True, text=True).stdout
    return out.startswith("True"), out.count("does not load")


def test_a_module_that_does_not_load_is_reported():
    from fovi_b200 import build
    assert build.build_native() == build.NATIVE
    assert imported_with("") == (True, 0)
    assert imported_with("sys.modules['fovi_b200._native'] = None") == (False, 1)
    other = "m = types.ModuleType('fovi_b200._native'); {}\nsys.modules['fovi_b200._native'] = m"
    assert imported_with(other.format("m.made_for = '0.1'")) == (False, 1)          # another torch
    assert imported_with(other.format("pass")) == (False, 1)                        # a module that does not say


@pytest.fixture
def made(monkeypatch, tmp_path):
    """build.build_native into a folder of its own, with a stand-in for the compiler that writes an empty file; the commands it was given."""
    from fovi_b200 import build
    commands = []

    def run(cmd, **kw):
        commands.append(cmd)
        open(cmd[cmd.index("-o") + 1], "w").close()
        return subprocess.CompletedProcess(cmd, 0, "", "")
    monkeypatch.setattr(build, "NATIVE", str(tmp_path / os.path.basename(build.NATIVE)))
    monkeypatch.setattr(build.subprocess, "run", run)
    return build, commands, tmp_path


def test_module_is_made_anew_for_another_torch(made, monkeypatch):
    build, commands, folder = made
    assert os.path.basename(build.NATIVE) == "_native" + sysconfig.get_config_var("EXT_SUFFIX")
    (folder / "_native.so").touch()                                       # any interpreter would import this one
    assert build.build_native() == build.build_native() == build.NATIVE and len(commands) == 1
    assert sorted(os.listdir(folder)) == sorted([os.path.basename(build.NATIVE), os.path.basename(build.NATIVE)[:-3] + ".stamp"])
    assert commands[0][commands[0].index("-o") + 1] != build.NATIVE       # not written in place
    torch, version = build._torch_version()
    monkeypatch.setattr(build, "_torch_version", lambda: (torch, version + ".other"))
    build.build_native()
    assert len(commands) == 2 and f'-DFOVI_TORCH_VERSION="{version}.other"' in commands[1]
    os.remove(build.NATIVE[:-3] + ".stamp")
    build.build_native()
    assert len(commands) == 3


@pytest.mark.parametrize("how", ["error", "no compiler"])
def test_a_module_that_cannot_be_made_leaves_the_python_path(made, monkeypatch, how):
    build, _, folder = made
    build.build_native()

    def fail(cmd, **kw):
        if how == "no compiler":
            raise FileNotFoundError(cmd[0])
        return subprocess.CompletedProcess(cmd, 1, "", "Python.h: no such file")
    monkeypatch.setattr(build.subprocess, "run", fail)
    with pytest.warns(UserWarning, match="not compiled"):
        assert build.build_native(force=True) is None
    assert os.listdir(folder) == []
