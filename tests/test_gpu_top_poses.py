"""The top-pose re-score beside the final keys, at the edges of its selection: k on both sides of
the short candidate list (8), fewer rotations than k, rotations that end inside and past a batch of
four per thread (1,024), and pairs re-scored together by the near-tie break."""
import numpy as np
import pytest

from cdocker_b200 import CDK_FORM_BF16X3, CDK_FORM_FP16X2, Receptor, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", [CDK_FORM_BF16X3, CDK_FORM_FP16X2])
@pytest.mark.parametrize("k,rots", [(1, 1), (8, 5), (8, 1023), (9, 257), (32, 31), (32, 1025), (8, 2049)])
def test_k_lowest(form, k, rots, grids_cache):
    w = synth.make_workload("c0_32", seed=7, n_conf=1, n_q=rots, grids_cache=grids_cache)
    with Receptor(w.grids, w.spacing, form=form, top_k=k) as rec:
        e, i = rec.search(w.coor, w.charge, w.eps, w.slot, w.quats)
        rot, te, tidx, e64 = rec.top_poses()
        assert rec.stats()["waves"] == 1
        m = min(k, rots)
        assert np.all(rot[m:] == -1) and len(set(rot[:m].tolist())) == m
        rot, te, tidx, e64 = rot[:m], te[:m], tidx[:m], e64[:m]
        assert np.array_equal(te, np.sort(e)[:m])  # ascending, the m smallest
        assert np.array_equal(te, e[rot]) and np.array_equal(tidx, i[rot])
        qq = w.quats.reshape(-1, 4)[rot]
        ref = rec.rescore_fp64(w.coor, w.charge, w.eps, w.slot, np.zeros(m, np.int32), qq, tidx)
    # two double sums of the same exact weights: 1e-7 is the bar of the oracle's float cells
    assert np.all(np.abs(e64 - ref) <= 1e-7 * np.maximum(1.0, np.abs(ref)))
