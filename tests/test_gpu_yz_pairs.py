"""The inverse (y,z) kernel over plane pairs against the single-plane kernels: the same bits, for
windows with odd and even edges in every dimension, one and many plane pairs per CTA, both B
layouts (FP32: pairs, one-column Hankel x pass: quads), and receptor grids holding infinities."""
import numpy as np
import pytest

from cdocker_b200 import CDK_FORM_BF16X3, CDK_FORM_FP16X2, CDK_FORM_FP32, Receptor

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", [CDK_FORM_FP32, CDK_FORM_FP16X2, CDK_FORM_BF16X3])
@pytest.mark.parametrize("n,rots,infinite", [(32, 300, False), (32, 1, True), (64, 67, False),
                                             (64, 3, True), (96, 40, False), (128, 1, False),
                                             (128, 33, False)])
def test_same_bits_as_single_planes(form, n, rots, infinite):
    rng = np.random.default_rng([n, rots])
    grids = rng.normal(size=(4, n, n, n)).astype(np.float32)
    if infinite:
        if form == CDK_FORM_FP16X2:
            pytest.skip("the scaled operator of an infinite grid has no FP16 form")
        grids[2, 1, 2, 3] = np.inf
    # boxes of 2 x 2.2 to 2 x 5.6 A axes: window edges n - 5 ... n - 24, of both parities
    atoms = 12
    coor = (rng.uniform(-1, 1, (1, atoms, 3)) * [5.6, 3.7, 2.2]).astype(np.float32)
    charge = rng.normal(0, 0.3, atoms).astype(np.float32)
    eps = rng.uniform(0.02, 0.2, atoms).astype(np.float32)
    slot = (np.arange(atoms) % 3).astype(np.int32)
    q = rng.normal(size=(rots, 4))
    q = (q / np.linalg.norm(q, axis=1, keepdims=True)).astype(np.float32)
    outs = []
    for kw in ({}, {"yz_block_stages": True}, {"yz_octets": True}):
        with Receptor(grids, 0.5, form=form, **kw) as rec:
            outs.append(rec.search(coor, charge, eps, slot, q[None]))
    for e, i in outs[1:]:
        np.testing.assert_array_equal(outs[0][1], i)
        np.testing.assert_array_equal(outs[0][0].view(np.uint32), e.view(np.uint32))
