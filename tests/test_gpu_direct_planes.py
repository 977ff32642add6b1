"""The direct plane kernel at the edges of its atom lists and chunks, against the FP64 oracle:
1 atom, counts around the 32-atom words, the largest ligand it takes (96 atoms), channels without
atoms, atoms on chunk borders, few rotations (several CTAs each) and many (one each)."""
import numpy as np
import pytest

from cdocker_b200 import CDK_FORM_BF16X3, CDK_FORM_FP16X2, CDK_FORM_FP32, Receptor
from oracle import oracle as O
from tests.parity import check_search

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form,tol", [(CDK_FORM_FP32, 1e-4), (CDK_FORM_FP16X2, 1e-3), (CDK_FORM_BF16X3, 1e-3)])
@pytest.mark.parametrize("n,atoms,rots", [(32, 1, 2), (32, 31, 3), (32, 32, 1000), (32, 33, 3), (32, 64, 4),
                                          (32, 65, 4), (32, 96, 5), (64, 96, 3), (96, 33, 2), (128, 65, 2)])
def test_atom_counts_vs_fp64(form, tol, n, atoms, rots):
    rng = np.random.default_rng([n, atoms])
    K = 5
    grids = rng.normal(size=(K, n, n, n)).astype(np.float32)
    # x on multiples of 4 A (borders of 8-plane chunks at 0.5 A) and between, slot 2 unused
    coor = rng.uniform(0, 3.5, (atoms, 3))
    coor[::3, 0] = 4.0 * rng.integers(0, 3, len(coor[::3]))
    coor = coor.astype(np.float32)[None]
    charge = rng.normal(0, 0.3, atoms).astype(np.float32)
    eps = rng.uniform(0.02, 0.2, atoms).astype(np.float32)
    slot = np.array([0, 1, 3])[rng.integers(0, 3, atoms)].astype(np.int32)
    q = rng.normal(size=(rots, 4))
    q[0] = [1, 0, 0, 0]
    q = (q / np.linalg.norm(q, axis=1, keepdims=True)).astype(np.float32)
    with Receptor(grids, 0.5, form=form) as rec:
        minE, idx = rec.search(coor, charge, eps, slot, q[None])
    some = np.arange(min(rots, 6)) * (rots - 1) // max(1, min(rots, 6) - 1)
    _, ridx, r64 = O.search_direct(grids, 0.5, coor, charge, eps, slot, q[some][None], prec=1)
    check_search(minE[some], idx[some], r64, ridx,
                 lambda r: O.energy_map(grids, 0.5, coor[0], charge, eps, slot, q[some[r]]), rel_tol=tol)


@pytest.mark.parametrize("n,atoms,rots,kw", [
    (32, 97, 3, {}), (32, 128, 131, {}), (32, 129, 3, {}), (64, 128, 2, {}), (64, 160, 2, {}),
    (64, 160, 2, {"tc_thread_copies": True}), (64, 110, 2, {"tc_thread_copies": True}),
    (96, 128, 2, {}), (128, 128, 1, {}), (128, 129, 1, {}), (32, 40, 130, {"fft_planes": True})])
def test_large_bf16_ligands_vs_fp64(n, atoms, rots, kw):
    """Split-BF16 ligands of 97 to 128 atoms (direct rows) and above (rows from FFT planes)."""
    rng = np.random.default_rng([n, atoms, 7])
    K = 4
    grids = rng.normal(size=(K, n, n, n)).astype(np.float32)
    coor = (rng.uniform(0, 1, (1, atoms, 3)) * [9.0, 7.0, 5.0]).astype(np.float32)
    charge = rng.normal(0, 0.3, atoms).astype(np.float32)
    eps = rng.uniform(0.02, 0.2, atoms).astype(np.float32)
    slot = rng.integers(0, K - 1, atoms).astype(np.int32)
    q = rng.normal(size=(rots, 4))
    q = (q / np.linalg.norm(q, axis=1, keepdims=True)).astype(np.float32)
    with Receptor(grids, 0.5, form=CDK_FORM_BF16X3, **kw) as rec:
        minE, idx = rec.search(coor, charge, eps, slot, q[None])
    some = np.arange(min(rots, 4)) * (rots - 1) // max(1, min(rots, 4) - 1)
    _, ridx, r64 = O.search_direct(grids, 0.5, coor, charge, eps, slot, q[some][None], prec=1)
    check_search(minE[some], idx[some], r64, ridx,
                 lambda r: O.energy_map(grids, 0.5, coor[0], charge, eps, slot, q[some[r]]), rel_tol=1e-3)
