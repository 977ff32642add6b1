"""The FP32 x pass at the edges of its launch shapes, against the FP64 oracle: ligand boxes on
both sides of every count of first-stage inputs (n/8 planes each), channels narrower than the
box, K from 2 to 16, rotation counts that fill no set of 4 and no chunk of 128."""
import numpy as np
import pytest

from cdocker_b200 import Receptor
from oracle import oracle as O
from tests.parity import check_search

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,K,box,rots,wave", [
    (32, 2, 6, 1, 0), (32, 9, 9, 5, 0), (32, 5, 14, 131, 0), (32, 16, 24, 6, 0),
    (64, 9, 15, 33, 7), (64, 3, 17, 3, 0), (64, 16, 26, 4, 0), (64, 9, 40, 3, 0),
    (96, 9, 24, 3, 0), (96, 4, 26, 2, 0), (96, 16, 40, 2, 0), (96, 2, 60, 2, 0),
    (128, 9, 17, 2, 0), (128, 2, 33, 2, 0), (128, 16, 50, 1, 0), (128, 16, 80, 1, 0),
])
def test_shapes_vs_fp64(n, K, box, rots, wave):
    rng = np.random.default_rng([n, K, box])
    grids = rng.normal(size=(K, n, n, n)).astype(np.float32)
    atoms = 3 * K
    v = rng.normal(size=(atoms, 3))
    # the first two atoms span the box, the others lie well inside it
    v = v / np.linalg.norm(v, axis=1, keepdims=True) * 0.25 * (box - 3) * rng.uniform(0.1, 0.9, (atoms, 1))
    v[:2] = [[0.25 * (box - 2.9), 0, 0], [-0.25 * (box - 2.9), 0, 0]]
    coor = v.astype(np.float32)[None]
    charge = rng.normal(0, 0.3, atoms).astype(np.float32)
    eps = rng.uniform(0.02, 0.2, atoms).astype(np.float32)
    slot = (np.arange(atoms) % (K - 1)).astype(np.int32)
    q = rng.normal(size=(rots, 4))
    q[0] = [1, 0, 0, 0]
    q = (q / np.linalg.norm(q, axis=1, keepdims=True)).astype(np.float32)
    with Receptor(grids, 0.5, wave_rotations=wave) as rec:
        minE, idx = rec.search(coor, charge, eps, slot, q[None])
        assert rec.stats()["box"] == box and rec.stats()["xpass_kind"] == "fp32_radix"
    _, ridx, r64 = O.search_direct(grids, 0.5, coor, charge, eps, slot, q[None], prec=1)
    check_search(minE, idx, r64, ridx,
                 lambda r: O.energy_map(grids, 0.5, coor[0], charge, eps, slot, q[r]))
