"""Searches from several threads, each on a context of its own whose launches ask for another amount of
dynamic shared memory (rotation counts and ligand boxes give the FP32 x pass other shapes, ligand sizes the
plane kernel, boxes the tensor-core x passes): every call succeeds with the bits of a call alone."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from cdocker_b200 import CDK_FORM_BF16X3, CDK_FORM_FP16X2, CDK_FORM_FP32, Receptor

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form,kw", [(CDK_FORM_FP32, {}), (CDK_FORM_FP16X2, {}), (CDK_FORM_BF16X3, {}),
                                     (CDK_FORM_BF16X3, {"tc_mma_sync": True})])
def test_shapes_of_other_threads(form, kw):
    n, K = 32, 9
    rng = np.random.default_rng(int(form))
    grids = rng.normal(size=(K, n, n, n)).astype(np.float32)

    def ligand(atoms, length, rots):
        q = rng.normal(size=(rots, 4))
        return ((rng.uniform(0, 1, (1, atoms, 3)) * [length, 3.0, 2.0]).astype(np.float32),
                rng.normal(0, 0.3, atoms).astype(np.float32), rng.uniform(0.02, 0.2, atoms).astype(np.float32),
                (np.arange(atoms) % (K - 1)).astype(np.int32),
                (q / np.linalg.norm(q, axis=1, keepdims=True)).astype(np.float32)[None])

    ligands = [ligand(*s) for s in ((8, 2.0, 3), (90, 5.0, 60), (24, 4.0, 700), (40, 6.0, 9),
                                    (12, 3.0, 330), (64, 7.0, 150))]

    def run(lig):
        bad = []
        with Receptor(grids, 0.5, form=form, **kw) as rec:
            first = rec.search(*lig)
            for _ in range(500):
                try:
                    got = rec.search(*lig)
                    if not all(np.array_equal(a, b) for a, b in zip(got, first)):
                        bad.append("other results")
                except Exception as e:
                    bad.append(str(e))
        return first, bad

    with Receptor(grids, 0.5, form=form, **kw) as rec:
        alone = [rec.search(*lig) for lig in ligands]
    with ThreadPoolExecutor(len(ligands)) as ex:
        outs = list(ex.map(run, ligands))
    for (first, bad), want in zip(outs, alone):
        assert not bad, bad[:3]
        for a, b in zip(first, want):
            np.testing.assert_array_equal(a, b)
