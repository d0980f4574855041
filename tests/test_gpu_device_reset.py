"""A context made after the process reset the device (cudaDeviceReset, which
ends the process's own device context and what was set in it) works as the
first one did."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CHILD = """
import ctypes, sys
sys.path[:0] = [{root!r}, {root!r} + "/oracle"]
import numpy as np
import torch                                   # brings libcudart.so.12 into the process
import oracle
from qld_b200 import api

rng = np.random.default_rng(3)
T = rng.integers(0, 1 << 63, (3000, 20), dtype=np.uint64)
bc, S = oracle.bitcounts(T), 20 * 64

def results():
    out = []
    with api.Context(0) as ctx:
        for mode in (api.R2_EXACT, api.R2_REFERENCE):
            ctx.set_option(api.OPT_R2_MODE, mode)
            for m in (300, 3000):              # tiles all at once; a few waves of tiles
                out += [ctx.ld(T[:m], bc[:m], S=S), *ctx.ld(T[:m], bc[:m], T[:m], bc[:m], S=S,
                                                            counts=True)]
        out.append(ctx.count_states(T[:200]))
    return out

first = results()
assert ctypes.CDLL("libcudart.so.12").cudaDeviceReset() == 0
again = results()
for m, (a, b) in zip((300, 300, 300, 3000, 3000, 3000) * 2 + (200,), zip(first, again)):
    keep = np.tri(m, dtype=bool).T             # what a single region owes, within any result
    assert np.array_equal(a[keep], b[keep], equal_nan=a.dtype == np.float32)
print("same")
"""


def test_context_after_device_reset():
    r = subprocess.run([sys.executable, "-c", CHILD.format(root=os.fspath(ROOT))], timeout=300,
                       capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.split()[-1] == "same", r.stderr[-2000:]
