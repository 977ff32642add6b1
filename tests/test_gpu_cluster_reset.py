"""Conformer selection across a reset of the process's own primary context: the memory kept between calls is
gone then, its address may be the caller's (it is, on a B200: the next allocation of the same size class gets
it), and neither a call nor a destroyed context may touch it."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import ctypes as C
import numpy as np
from cdocker_b200 import Receptor, synth
from cdocker_b200.conformers import cluster_conformers
cu = C.CDLL("libcuda.so.1")
dev, ctx = C.c_int(), C.c_void_p()
x, e = synth.conformer_ensemble(3, n_atoms=20, n_conf=200, n_rotors=4)
want = cluster_conformers(x, e, 1.5, 50)
assert cu.cuDeviceGet(C.byref(dev), 0) == 0
for release in (False, True):
    assert cu.cuDevicePrimaryCtxReset_v2(dev) == 0
    assert cu.cuDevicePrimaryCtxRetain(C.byref(ctx), dev) == 0 and cu.cuCtxSetCurrent(ctx) == 0
    mine = []
    for _ in range(24):  # the caller's own memory, over the addresses that were kept
        p = C.c_uint64()
        assert cu.cuMemAlloc_v2(C.byref(p), C.c_size_t(1 << 20)) == 0
        assert cu.cuMemsetD8_v2(p, C.c_ubyte(0x5a), C.c_size_t(1 << 20)) == 0
        mine.append(p)
    if release:  # a context's end gives kept memory back
        Receptor(np.zeros((2, 32, 32, 32), np.float32), 0.5).close()
    got = cluster_conformers(x, e, 1.5, 50)
    assert np.array_equal(got, want)
    host = np.empty(1 << 20, np.uint8)
    for p in mine:
        assert cu.cuMemcpyDtoH_v2(host.ctypes.data_as(C.c_void_p), p, C.c_size_t(1 << 20)) == 0
        assert np.all(host == 0x5a), "a conformer call wrote into the caller's memory"
    assert cu.cuDevicePrimaryCtxRelease_v2(dev) == 0
print("ok")
"""


def test_selection_after_a_reset_leaves_the_callers_memory_alone():
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, PYTHONPATH=ROOT))
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
