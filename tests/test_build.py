"""The build of the two shared libraries, with compilers that only write a file: what is linked to what, when a module is built
anew, and that processes which build at the same time do it once and never meet half a file."""
import os
import shutil
import subprocess
import sys
import time

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = "flashnystrom_b200"
WHOLE = "first half, second half"

_COMPILER = f"""#!/bin/sh
echo "$(basename "$0") $*" >> "$BUILD_LOG"
while [ "$1" != "-o" ]; do shift; done
printf 'first half, ' > "$2"
sleep 0.4
printf 'second half' >> "$2"
"""


@pytest.fixture
def tree(tmp_path):
    """A copy of the tree with what the build reads; run(code) starts Python in it with `build` imported."""
    (tmp_path / PKG / "csrc").mkdir(parents=True)
    (tmp_path / "include").mkdir()
    shutil.copy(os.path.join(ROOT, PKG, "build.py"), tmp_path / PKG)
    shutil.copy(os.path.join(ROOT, PKG, "csrc", "native.cpp"), tmp_path / PKG / "csrc")
    shutil.copy(os.path.join(ROOT, "include", "flashnystrom_b200.h"), tmp_path / "include")
    (tmp_path / PKG / "csrc" / "fnb_api.cu").write_text("")
    (tmp_path / "bin").mkdir()
    for name in ("nvcc", "cxx"):
        (tmp_path / "bin" / name).write_text(_COMPILER)
        (tmp_path / "bin" / name).chmod(0o755)

    class Tree:
        log, lib = tmp_path / "log", tmp_path / PKG / "lib"
        header = tmp_path / "include" / "flashnystrom_b200.h"

        def start(self, code, **more):
            env = dict(os.environ, PATH=f"{tmp_path / 'bin'}:{os.environ['PATH']}", CXX=str(tmp_path / "bin" / "cxx"), BUILD_LOG=str(self.log))
            env.update(more)
            return subprocess.Popen([sys.executable, "-c", f"import sys; sys.path.insert(0, {str(tmp_path / PKG)!r}); import torch, build; {code}"], env=env)

        def run(self, code, **env):
            assert self.start(code, **env).wait(120) == 0

        def compiled(self):
            return [line.split()[0] for line in self.log.read_text().splitlines()]

        def modules(self):
            return sorted(p.name for p in self.lib.glob("_native*"))
    return Tree()


def test_processes_at_the_same_time_build_once(tree):
    processes = [tree.start("build.build()") for _ in range(3)]
    while any(p.poll() is None for p in processes):
        for path in tree.lib.glob("*.so"):
            if ".part" not in path.name:
                assert path.read_text() == WHOLE, path
        time.sleep(0.01)
    assert [p.returncode for p in processes] == [0, 0, 0]
    assert tree.compiled() == ["nvcc", "cxx"]
    assert len(tree.modules()) == 1 and not list(tree.lib.glob("*.part*"))


def test_module_is_never_linked_to_a_variant(tree):
    tree.run("build.build()", FNB_LIB_NAME="variant.so")
    assert [p.name for p in tree.lib.iterdir()] == ["variant.so"]
    tree.run("build.build_native()", FNB_LIB_NAME="variant.so")
    link = tree.log.read_text().splitlines()[-1].split()
    assert "-l:libflashnystrom_b200.so" in link and "-l:variant.so" not in link
    assert (tree.lib / "libflashnystrom_b200.so").exists()


def test_module_follows_header_and_torch(tree):
    tree.run("build.build(); build.build()")
    first = tree.modules()
    assert tree.compiled() == ["nvcc", "cxx"]
    tree.run("torch.__version__ = '9.9'; build.build()")           # (another torch's module stays where it is)
    assert len(tree.modules()) == 2 and set(first) < set(tree.modules())
    tree.header.write_text(tree.header.read_text() + "\n// one line more\n")
    os.utime(tree.header, (0, 0))                                  # (however old the file looks)
    tree.run("build.build()")
    assert len(tree.modules()) == 2 and not set(first) & set(tree.modules())
    assert tree.compiled() == ["nvcc", "cxx", "cxx", "cxx"]


def test_a_failed_build_leaves_nothing(tree):
    tree.run("build.build_library()")
    assert tree.start("build.build_native()", CXX="false").wait(120) != 0
    assert not tree.modules()


def test_the_package_loads_the_module_that_the_build_names():
    from flashnystrom_b200 import _lib, build
    assert _lib.native().__file__ == build.native_path()
    assert _lib.LIB_PATH == build.PACKAGE_LIB
