"""The stacking of downloaded columns (pydsmc.gpu._rows): np.stack's values on
either side of its threads' parts (65,536 rows), also while the interpreter
exits, when a solver's last download may still run."""
import os
import subprocess
import sys

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
