"""The stacking of downloaded columns (pydsmc.gpu._rows): np.stack's values on
either side of its threads' parts (65,536 rows), also from several threads at
once, where no thread can be had, in a forked process, and while the
interpreter exits, when a solver's last download may still run."""
import os
import subprocess
import sys
import threading

import numpy as np
import pytest

from pydsmc import gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("n", [0, 1, 65535, 65536, 65537, 131072, 700001])
def test_rows_is_np_stack(n):
    cols = [np.random.default_rng(k).random(n) for k in range(3)]
    got = gpu._rows(cols)
    want = np.stack(cols, 1)
    assert got.dtype == want.dtype and got.flags["C_CONTIGUOUS"] and np.array_equal(got, want)


def test_rows_at_interpreter_exit():
    code = ("import atexit, numpy as np\n"
            "from pydsmc import gpu\n"
            "c = [np.arange(200001.0) + k for k in range(3)]\n"
            "gpu._rows(c)\n"
            "atexit.register(lambda: print(bool(np.array_equal(gpu._rows(c), np.stack(c, 1)))))\n")
    env = dict(os.environ, PYTHONPATH=os.path.join(ROOT, "dig-appolo_b200"))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=120, env=env)
    assert r.returncode == 0 and r.stdout.strip() == "True", r.stdout + r.stderr


def test_rows_without_threads(monkeypatch):
    def none(*a, **k):
        raise RuntimeError("can't start new thread")
    cols = [np.arange(300001.0) + k for k in range(3)]
    monkeypatch.setattr(gpu, "_rows_pool", None)
    monkeypatch.setattr(threading.Thread, "start", none)
    assert np.array_equal(gpu._rows(cols), np.stack(cols, 1))


def test_rows_from_several_threads():
    cols = [[np.random.default_rng(10 * j + k).random(200001) for k in range(3)] for j in range(6)]
    got = [None] * 6
    jobs = [threading.Thread(target=lambda j=j: got.__setitem__(j, gpu._rows(cols[j]))) for j in range(6)]
    for t in jobs:
        t.start()
    for t in jobs:
        t.join()
    assert all(np.array_equal(g, np.stack(c, 1)) for g, c in zip(got, cols))


def test_rows_in_a_forked_process():
    code = ("import os, numpy as np\n"
            "from pydsmc import gpu\n"
            "c = [np.arange(200001.0) + k for k in range(3)]\n"
            "gpu._rows(c)\n"
            "pid = os.fork()\n"
            "if pid == 0:\n"
            "    os._exit(0 if np.array_equal(gpu._rows(c), np.stack(c, 1)) else 1)\n"
            "print(os.waitstatus_to_exitcode(os.waitpid(pid, 0)[1]) == 0)\n")
    env = dict(os.environ, PYTHONPATH=os.path.join(ROOT, "dig-appolo_b200"))
    r = subprocess.run([sys.executable, "-W", "ignore", "-c", code], capture_output=True, text=True, timeout=120, env=env)
    assert r.returncode == 0 and r.stdout.strip() == "True", r.stdout + r.stderr
