"""The largest search that the caller-owned-memory entry point's 64 MiB hold to the byte: one rotation at 128^3,
K = 16, a box of 55 planes, with a conformer table that leaves no 16 bytes over."""
import ctypes as C

import numpy as np
import pytest

from cdocker_b200 import Receptor
from cdocker_b200 import _lib as L

pytestmark = pytest.mark.gpu


def test_a_search_that_fills_the_scratch():
    import torch
    n, K, atoms, confs = 128, 16, 52, 784
    rng = np.random.default_rng(4)
    grids = rng.normal(size=(K, n, n, n)).astype(np.float32)
    v = rng.uniform(-3, 3, (atoms, 3))
    v[:2] = [[13.1, 0, 0], [-13.1, 0, 0]]  # 26.2 A: 55 planes
    q = rng.normal(size=(confs, 1, 4))
    lig = (np.repeat(v.astype(np.float32)[None], confs, 0), rng.normal(0, 0.3, atoms).astype(np.float32),
           rng.uniform(0.02, 0.2, atoms).astype(np.float32), (np.arange(atoms) % (K - 1)).astype(np.int32),
           (q / np.linalg.norm(q, axis=-1, keepdims=True)).astype(np.float32))
    dev = [torch.from_numpy(a).cuda() for a in lig]
    e = torch.empty(confs, dtype=torch.float32, device="cuda")
    i = torch.empty(confs, 3, dtype=torch.int32, device="cuda")
    with Receptor(grids, 0.5) as rec:
        want = rec.search(*lig)
        assert rec.stats()["box"] == 55
        L.check(L.lib().cdk_search_device_noalloc(
            rec.handle, atoms, confs, *(C.c_void_p(t.data_ptr()) for t in dev[:4]), 1,
            C.c_void_p(dev[4].data_ptr()), C.c_void_p(e.data_ptr()), C.c_void_p(i.data_ptr()), None))
    np.testing.assert_array_equal(i.cpu().numpy(), want[1])
    np.testing.assert_array_equal(e.cpu().numpy().view(np.uint32), want[0].view(np.uint32))
