"""The Makefile's rules for the torch extension, run on a copy of the sources with stand-ins for Python and the
compilers: the C-ABI library needs no torch, a probe that fails leaves nothing behind, and another torch means a
rebuild."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CALL = "../_torch_call.fake-abi.so"


@pytest.fixture
def tree(tmp_path):
    csrc = tmp_path / "kermac_b200" / "csrc"
    shutil.copytree(os.path.join(ROOT, "kermac_b200", "csrc"), csrc, ignore=shutil.ignore_patterns("build", "__pycache__"))
    shutil.copytree(os.path.join(ROOT, "include"), tmp_path / "include")
    # compilers that write their command line to their output file
    for name in ("cxx", "nvcc"):
        tool = tmp_path / name
        tool.write_text('#!/bin/sh\nall="$*"\nwhile [ $# -gt 0 ]; do [ "$1" = -o ] && out="$2"; shift; done\n'
                        f'echo "$all" > "$out"\necho "$all" >> {tmp_path}/{name}.log\n')
        tool.chmod(0o755)
    return tmp_path


def _python(tree, version, fails_on="nothing"):
    fake = tree / "python"
    fake.write_text(f'#!/bin/sh\n[ "$2" = {fails_on} ] && exit 1\ncase "$2" in\n  id) echo "torch {version}" ;;\n'
                    f'  suffix) echo .fake-abi.so ;;\n  *) echo "-Dflag_{version}" ;;\nesac\n')
    fake.chmod(0o755)
    return str(fake)


def _make(tree, python, *targets):
    return subprocess.run(["make", "-C", str(tree / "kermac_b200" / "csrc"), f"PYTHON={python}", f"CXX={tree}/cxx",
                           f"NVCC={tree}/nvcc", *targets], capture_output=True, text=True)


def _compiled(tree, name):
    log = tree / f"{name}.log"
    return log.read_text().splitlines() if log.exists() else []


@pytest.mark.parametrize("target", [["../libkermac_b200.so"], []])
def test_the_library_is_built_without_torch(tree, target):
    run = _make(tree, "false", *target)
    assert run.returncode == 0, run.stderr
    assert (tree / "kermac_b200" / "libkermac_b200.so").exists()
    assert not _compiled(tree, "cxx") and not list((tree / "kermac_b200" / "csrc" / "build").glob("torch*"))
    run = _make(tree, "false", "../_torch_call")            # (no Python, no file name ending)
    assert run.returncode != 0 and "needs torch" in run.stderr


def test_a_probe_that_fails_is_repeated(tree):
    assert _make(tree, _python(tree, "1.0", fails_on="cflags"), CALL).returncode != 0
    assert not _compiled(tree, "cxx")
    assert _make(tree, _python(tree, "1.0"), CALL).returncode == 0
    assert any("-Dflag_1.0" in line for line in _compiled(tree, "cxx"))


def test_the_extension_is_rebuilt_for_another_torch_only(tree):
    for version, expected in (("1.0", 2), ("1.0", 2), ("1.1", 4)):      # one compilation and one link each time
        run = _make(tree, _python(tree, version), CALL)
        assert run.returncode == 0, run.stderr
        lines = _compiled(tree, "cxx")
        assert len(lines) == expected and any(f"-Dflag_{version}" in line for line in lines[-2:])
