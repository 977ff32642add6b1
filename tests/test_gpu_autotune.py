"""What the autotuner may choose: never a shape that makes the search slower than without it. FP32: from 256
rotations on the plan's own rotations per CTA, also after a smaller search has tuned the box; tensor-core forms:
not two columns per CTA where the inverse pass loses more than the x pass gains; timing runs leave the work
counters alone."""
import numpy as np
import pytest

from cdocker_b200 import CDK_FORM_FP16X2, Receptor

pytestmark = pytest.mark.gpu


def workload(n, K, rots):
    rng = np.random.default_rng([n, K])
    grids = rng.normal(size=(K, n, n, n)).astype(np.float32)
    v = rng.normal(size=(24, 3))
    coor = (v / np.linalg.norm(v, axis=1, keepdims=True) * 2.2).astype(np.float32)[None]
    q = rng.normal(size=(rots, 4))
    return grids, (coor, rng.normal(0, 0.3, 24).astype(np.float32), rng.uniform(0.02, 0.2, 24).astype(np.float32),
                   (np.arange(24) % (K - 1)).astype(np.int32),
                   (q / np.linalg.norm(q, axis=1, keepdims=True)).astype(np.float32)[None])


@pytest.mark.parametrize("n,rots", [(32, 256), (32, 2000), (64, 700), (96, 300)])
def test_fp32_keeps_the_plan(n, rots):
    grids, lig = workload(n, 9, rots)
    with Receptor(grids, 0.5) as rec:
        want = rec.search(*lig)
        chunk = rec.stats()["rotations_per_cta"]
    with Receptor(grids, 0.5, autotune=True) as rec:
        small = rec.search(*lig[:4], lig[4][:, :40])
        got = rec.search(*lig)
        assert rec.stats()["rotations_per_cta"] == chunk
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)
    for a, b in zip(small, want):
        np.testing.assert_array_equal(a, b[:40])


def test_hankel_counts_the_inverse_pass():
    grids, lig = workload(32, 3, 20000)
    out = []
    for autotune in (False, True):
        with Receptor(grids, 0.5, form=CDK_FORM_FP16X2, autotune=autotune) as rec:
            out.append((rec.search(*lig), rec.stats()))
    (want, st0), (got, st1) = out
    assert st1["col_tile"] == 1
    for key in ("tensor_steps", "mma_units", "planes_spread", "planes_window"):
        assert st1[key] == st0[key]
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)
