"""Building the native extension: an interrupted build must never make a later one wait for ever, and a
wait for a build that is going on has a limit.  A one-line extension stands in for the real sources."""
import os
import signal
import subprocess
import sys
import textwrap
import time
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
SOURCE = """
#include <Python.h>
static PyModuleDef def = {PyModuleDef_HEAD_INIT, "pccl_C"};
PyMODINIT_FUNC PyInit_pccl_C() {
  PyObject* m = PyModule_Create(&def);
  PyModule_AddIntConstant(m, "answer", 42);
  return m;
}
"""
# builds in the directory given as the first argument and prints what the module holds
BUILDER = """
import os, sys, time
sys.path.insert(0, {root!r})
from pathlib import Path
from pccl import build_kernels as bk
work = Path(sys.argv[1])
bk.CSRC, bk.BUILD_DIR, bk.SOURCES = work / "csrc", work / "_build", ["one.cpp"]
bk._SO, bk._DIGEST = bk.BUILD_DIR / "pccl_C.so", bk.BUILD_DIR / "pccl_C.digest"
bk._LOCK = bk.BUILD_DIR / "pccl_C.lock"
bk.NVCC_FLAGS = []
print("building", flush=True)
print("answer", bk.build().answer, flush=True)
"""


@pytest.fixture
def tree(tmp_path):
    (tmp_path / "csrc").mkdir()
    (tmp_path / "csrc" / "one.cpp").write_text(SOURCE)
    (tmp_path / "builder.py").write_text(textwrap.dedent(BUILDER).format(root=str(ROOT)))
    return tmp_path


def run_builder(tree, timeout=90, **env):
    return subprocess.run([sys.executable, str(tree / "builder.py"), str(tree)], capture_output=True, text=True,
                          timeout=timeout, env={**os.environ, **env})


def finished(tree):
    out = run_builder(tree)
    assert out.returncode == 0 and "answer 42" in out.stdout, out.stderr[-2000:]
    assert (tree / "_build" / "pccl_C.so").exists() and (tree / "_build" / "pccl_C.digest").exists()


@pytest.mark.parametrize("where", ["_build", "_build/obj"])
def test_a_lock_file_without_a_holder_is_no_obstacle(tree, where):
    (tree / where).mkdir(parents=True)
    (tree / where / "lock").touch()
    (tree / "_build" / "pccl_C.lock").touch()
    finished(tree)
    finished(tree)                       # and the second call finds it built


def test_a_killed_build_is_begun_again_by_the_next_call(tree):
    slow = tree / "slow"
    slow.mkdir()
    (slow / "g++").write_text("#!/bin/sh\ntouch %s/compiling\nsleep 60\nexec /usr/bin/g++ \"$@\"\n" % tree)
    (slow / "g++").chmod(0o755)
    p = subprocess.Popen([sys.executable, str(tree / "builder.py"), str(tree)], start_new_session=True,
                         env={**os.environ, "PCCL_KEEP_COMPILER": "1", "CXX": str(slow / "g++")})
    try:
        deadline = time.monotonic() + 60
        while not (tree / "compiling").exists():
            assert time.monotonic() < deadline and p.poll() is None
            time.sleep(0.05)
    finally:
        os.killpg(p.pid, signal.SIGKILL)
        p.wait()
    assert not (tree / "_build" / "pccl_C.digest").exists()
    finished(tree)


def test_a_wait_for_another_build_ends_with_an_error_that_names_the_lock(tree):
    import fcntl

    (tree / "_build").mkdir()
    with open(tree / "_build" / "pccl_C.lock", "w") as f:
        fcntl.flock(f, fcntl.LOCK_EX)
        out = run_builder(tree, PCCL_BUILD_WAIT_S="0.5")
    assert out.returncode != 0 and "TimeoutError" in out.stderr and "pccl_C.lock" in out.stderr
    finished(tree)
