"""Split-BF16 searches off the direct plane path (ligands above 96 atoms, planes by the FFT): the same bits and
the same kind as the x pass that such ligands always had, in-kernel operand builds at 64^3 and mma.sync
at the other grids, whatever the number of rotations."""
import numpy as np
import pytest

from cdocker_b200 import CDK_FORM_BF16X3, Receptor

pytestmark = pytest.mark.gpu


def search(n, K, atoms, rots, length=9.0, **kw):
    rng = np.random.default_rng([n, atoms])
    grids = rng.normal(size=(K, n, n, n)).astype(np.float32)
    coor = (rng.uniform(0, 1, (1, atoms, 3)) * [length, 7.0, 5.0]).astype(np.float32)
    charge = rng.normal(0, 0.3, atoms).astype(np.float32)
    eps = rng.uniform(0.02, 0.2, atoms).astype(np.float32)
    slot = rng.integers(0, K - 1, atoms).astype(np.int32)
    q = rng.normal(size=(2000, 4))
    q = (q / np.linalg.norm(q, axis=1, keepdims=True)).astype(np.float32)[None, :rots]
    with Receptor(grids, 0.5, form=CDK_FORM_BF16X3, **kw) as rec:
        minE, idx = rec.search(coor, charge, eps, slot, q)
        return minE, idx, rec.stats()["xpass_kind"]


@pytest.mark.parametrize("n,K,atoms,rots,kw", [
    (32, 9, 97, 40, {}), (64, 9, 100, 300, {}), (64, 2, 97, 1, {}), (64, 9, 128, 130, {}), (96, 9, 110, 3, {}),
    (128, 4, 97, 2, {}), (64, 9, 110, 40, {"tc_hankel": True}), (32, 4, 129, 3, {}), (64, 9, 129, 200, {}), (64, 3, 250, 1, {}), (96, 4, 160, 5, {}), (128, 3, 129, 2, {}),
    (32, 4, 40, 150, {"fft_planes": True}), (64, 9, 40, 30, {"fft_planes": True})])
def test_same_x_pass_as_asked_for(n, K, atoms, rots, kw):
    other = {"tc_build": True} if n == 64 else {"tc_mma_sync": True}
    e, i, kind = search(n, K, atoms, rots, **kw)
    we, wi, wkind = search(n, K, atoms, rots, **kw, **other)
    assert kind == wkind == ("tcgen05_build" if n == 64 else "mma_sync")
    np.testing.assert_array_equal(i, wi)
    np.testing.assert_array_equal(e.view(np.uint32), we.view(np.uint32))
