"""Calls of the network's C entry points whose arrays fit no memory are refused
with an error status: no exception leaves them.  In a process of its own, which
an exception out of a C function would end."""
import subprocess
import sys

import pytest

from conftest import ROOT

CALL = """
import ctypes, sys
sys.path.insert(0, {root!r})
import numpy as np
from cl_forward_gb300 import build, native
build.build()
lib = native.load()
a = np.zeros(native.MLP_PARAMS + 100, np.float32)
p = a.ctypes.data_as(ctypes.c_void_p)
status = {call}
assert status not in (native.OK, -1), status
print("refused", status)
"""


@pytest.mark.parametrize("call", [
    "lib.velo_mlp_train(p, p, p, 10, 2 ** 31 - 1, 2 ** 31 - 1, 1e-3, 1, p, None)",
    "lib.velo_mlp_train(p, p, p, 2 ** 62, 3, 10, 1e-3, 1, p, None)",
    "lib.velo_mlp_grad(p, p, p, p, 2 ** 62, p, None)",
    "lib.velo_mlp_forward(p, p, 2 ** 62, p)"])
def test_too_large(native_lib, call):
    r = subprocess.run([sys.executable, "-c", CALL.format(root=ROOT, call=call)], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and "refused" in r.stdout, (r.returncode, r.stdout, r.stderr)
