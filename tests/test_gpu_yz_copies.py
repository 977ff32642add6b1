"""The inverse (y,z) kernels with bulk copies (two plane pairs at once at n <= 64, one FP32 pair
above) against the single-plane kernel: the same bits, with one turn per CTA (few rotations) and
several (many), for windows that leave 1, 2, 3 or 4 planes in the last quad, with and without the two
smallest keys."""
import numpy as np
import pytest

from cdocker_b200 import CDK_FORM_BF16X3, CDK_FORM_FP16X2, CDK_FORM_FP32, Receptor

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", [CDK_FORM_FP32, CDK_FORM_FP16X2, CDK_FORM_BF16X3])
@pytest.mark.parametrize("tie_break", [True, False])
@pytest.mark.parametrize("n,rots,atoms", [(32, 2, 5), (32, 2500, 9), (64, 3, 40), (64, 900, 14),
                                          (96, 1, 9), (96, 250, 14), (128, 160, 9)])
def test_same_bits_as_single_planes(form, tie_break, n, rots, atoms):
    rng = np.random.default_rng([n, rots, atoms])
    grids = rng.normal(size=(3, n, n, n)).astype(np.float32)
    coor = (rng.uniform(-1, 1, (1, atoms, 3)) * [4.9, 2.8, 1.4]).astype(np.float32)
    charge = rng.normal(0, 0.3, atoms).astype(np.float32)
    eps = rng.uniform(0.02, 0.2, atoms).astype(np.float32)
    slot = (np.arange(atoms) % 2).astype(np.int32)
    q = rng.normal(size=(rots, 4))
    q = (q / np.linalg.norm(q, axis=1, keepdims=True)).astype(np.float32)
    outs = []
    for kw in ({}, {"yz_octets": True}):
        with Receptor(grids, 0.5, form=form, tie_break=tie_break, **kw) as rec:
            outs.append(rec.search(coor, charge, eps, slot, q[None]))
    np.testing.assert_array_equal(outs[0][1], outs[1][1])
    np.testing.assert_array_equal(outs[0][0].view(np.uint32), outs[1][0].view(np.uint32))
