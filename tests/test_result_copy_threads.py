"""The binding's copy of large results where its threads are not to be had: in an exit handler, and in a child process
forked after they were started (CPU)."""
import subprocess
import sys

import pytest

_HEAD = """
import sys
sys.path[:0] = {paths!r}
import atexit, os, signal
import numpy as np
import fastbc_gpu as fg
a = np.arange(3_000_001, dtype=np.float64)
"""


@pytest.mark.parametrize("body", [
    "atexit.register(lambda: print(np.array_equal(fg._copy(a), a)))",
    "fg._copy(a); atexit.register(lambda: print(np.array_equal(fg._copy(a), a)))",
    "fg._copy(a)\npid = os.fork()\nif pid == 0:\n    signal.alarm(20)\n    print(np.array_equal(fg._copy(a), a), flush=True)\n"
    "    os._exit(0)\nassert os.waitpid(pid, 0)[1] == 0"])
def test_without_threads(body):
    out = subprocess.run([sys.executable, "-c", _HEAD.format(paths=sys.path[:4]) + body], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout.split() == ["True"], out.stderr
