"""Precision-form servers on waves that the tensor-core x pass does not take: ligands above 96 atoms,
ligand boxes above 32 planes, receptors set to another tensor-core kernel, K x n without a Hankel
shape. Such waves run the FP32 x pass with the FP64 near-tie break: against the FP64 oracle, and bit
for bit the FP32 form's energies where the translation is the same; small requests of the same wave
succeed with them."""
import numpy as np
import pytest

from cdocker_b200 import CDK_FORM_BF16X3, CDK_FORM_FP16X2, Receptor
from cdocker_b200.serving import Server
from oracle import oracle as O
from tests.parity import check_search

pytestmark = pytest.mark.gpu


def _request(rng, K, atoms, box, rots):
    """A ligand whose first two atoms span `box` planes of 0.5 A and whose others lie inside."""
    v = rng.normal(size=(atoms, 3))
    v = v / np.linalg.norm(v, axis=1, keepdims=True) * 0.25 * (box - 3) * rng.uniform(0.1, 0.9, (atoms, 1))
    v[:2] = [[0.25 * (box - 2.9), 0, 0], [-0.25 * (box - 2.9), 0, 0]]
    q = rng.normal(size=(rots, 4))
    q = (q / np.linalg.norm(q, axis=1, keepdims=True)).astype(np.float32)
    return (v.astype(np.float32)[None], rng.normal(0, 0.3, atoms).astype(np.float32),
            rng.uniform(0.02, 0.2, atoms).astype(np.float32),
            (np.arange(atoms) % (K - 1)).astype(np.int32), q[None])


@pytest.mark.parametrize("form", [CDK_FORM_BF16X3, CDK_FORM_FP16X2])
@pytest.mark.parametrize("n,K,sizes,kw", [
    (32, 5, ((110, 20, 70),), {}), (64, 5, ((97, 20, 9), (12, 8, 200)), {}),
    (64, 4, ((20, 36, 40), (30, 12, 30)), {}), (96, 3, ((128, 24, 5), (9, 10, 6)), {}),
    (128, 3, ((100, 20, 3),), {}), (128, 16, ((30, 12, 2),), {}),
    (64, 5, ((20, 12, 30),), {"tc_mma_sync": True}), (64, 5, ((20, 12, 30),), {"tc_build": True}),
    (64, 5, ((20, 12, 30),), {"fft_planes": True}), (64, 5, ((110, 20, 30),), {"tie_break": False}),
])
def test_fallback_waves(form, n, K, sizes, kw):
    if form == CDK_FORM_FP16X2 and (kw.get("tc_mma_sync") or kw.get("tc_build")):
        pytest.skip("the split-FP16 form serves tensor-core waves whatever kernel is asked for")
    rng = np.random.default_rng([n, K, len(sizes)])
    grids = rng.normal(size=(K, n, n, n)).astype(np.float32)
    reqs = [_request(rng, K, *s) for s in sizes]
    with Receptor(grids, 0.5, form=form, **kw) as rec:
        with Server(rec, arena_bytes=16 << 20, wave_rotations=256, max_box=40 if n > 40 else n) as srv:
            tickets = [srv.submit(*r) for r in reqs]
            got = [srv.poll(t, -1) for t in tickets]
            st = srv.stats()
    assert st["tc_waves"] < st["waves"] and st["completed"] == len(reqs)
    with Receptor(grids, 0.5, fft_planes=kw.get("fft_planes", False)) as rec:  # the same ligand planes
        fp32 = [rec.search(*r) for r in reqs]
    # the first request never shares a wave that the tensor cores take
    e, i, _ = got[0]
    same = np.all(i == fp32[0][1], axis=1)
    assert same.mean() >= 0.9
    np.testing.assert_array_equal(e[same].view(np.uint32), fp32[0][0][same].view(np.uint32))
    for (e, i, _), (coor, charge, eps, slot, quats) in zip(got, reqs):
        q = quats[0]
        _, ridx, r64 = O.search_direct(grids, 0.5, coor, charge, eps, slot, quats, prec=1)
        check_search(e, i, r64, ridx, lambda r: O.energy_map(grids, 0.5, coor[0], charge, eps, slot, q[r]),
                     rel_tol=1e-3)
