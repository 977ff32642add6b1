"""The FP32 x pass on both sides of the rule that takes waves of a few rotations and the largest boxes at 128^3
to the block-stage kernel: the same bits whatever the number of rotations searched with a rotation, from plain
searches, the caller-owned-memory search and a server; and the FP64 oracle for a box on each side."""
import ctypes as C

import numpy as np
import pytest

from cdocker_b200 import Receptor
from cdocker_b200 import _lib as L
from cdocker_b200.serving import Server
from oracle import oracle as O
from tests.parity import check_search

pytestmark = pytest.mark.gpu


def workload(n, K, box, rots):
    rng = np.random.default_rng([n, K, box])
    grids = rng.normal(size=(K, n, n, n)).astype(np.float32)
    atoms = 3 * K
    v = rng.normal(size=(atoms, 3))
    # the first two atoms span the box, the others lie well inside it
    v = v / np.linalg.norm(v, axis=1, keepdims=True) * 0.25 * (box - 3) * rng.uniform(0.1, 0.9, (atoms, 1))
    v[:2] = [[0.25 * (box - 2.9), 0, 0], [-0.25 * (box - 2.9), 0, 0]]
    q = rng.normal(size=(rots, 4))
    return grids, (v.astype(np.float32)[None], rng.normal(0, 0.3, atoms).astype(np.float32),
                   rng.uniform(0.02, 0.2, atoms).astype(np.float32), (np.arange(atoms) % (K - 1)).astype(np.int32),
                   (q / np.linalg.norm(q, axis=1, keepdims=True)).astype(np.float32)[None])


def same(got, want, count):
    np.testing.assert_array_equal(got[1], want[1][:count])
    np.testing.assert_array_equal(got[0].view(np.uint32), want[0][:count].view(np.uint32))


# most rotations of the block-stage kernel for boxes up to n/2 and above
@pytest.mark.parametrize("n,K,box,most", [
    (32, 2, 9, 5), (32, 9, 24, 3), (64, 2, 10, 5), (64, 9, 21, 5), (64, 16, 40, 7), (96, 3, 20, 5), (96, 9, 70, 15),
    (96, 12, 60, 24), (128, 2, 17, 3), (128, 9, 75, 8), (128, 2, 100, 8)])
def test_bits_do_not_depend_on_the_number_of_rotations(n, K, box, most):
    grids, lig = workload(n, K, box, 40)
    with Receptor(grids, 0.5) as rec:
        want = rec.search(*lig)
        assert rec.stats()["col_tile"] == 8
        for count in sorted({1, 2, most - 1, most, most + 1, most + 2}):
            got = rec.search(*lig[:4], lig[4][:, :count])
            st = rec.stats()
            assert st["xpass_kind"] == "fp32_radix"
            if count <= most or K < 12:  # the other kernel's plan may come to 32 as well with two groups of warps
                assert (st["rotations_per_cta"] == 32) == (count <= most)
            same(got, want, count)
        with Server(rec, arena_bytes=1 << 22, wave_rotations=64, max_box=n, max_atoms=64) as srv:
            e, i, _ = srv.poll(srv.submit(*lig[:4], lig[4][:, :2]), -1)
            same((e, i), want, 2)


@pytest.mark.parametrize("K,box", [(5, 80), (5, 86), (9, 100), (12, 88), (12, 96), (16, 120)])
def test_largest_boxes_at_128(K, box):
    grids, lig = workload(128, K, box, 10)
    with Receptor(grids, 0.5) as rec:
        got = rec.search(*lig)
        assert (rec.stats()["rotations_per_cta"] == 32) == (box > (80 if K < 10 else 88))
    with Receptor(grids, 0.5, wave_rotations=9) as rec:  # a last wave of one rotation
        same(rec.search(*lig), got, 10)
    _, ridx, r64 = O.search_direct(grids, 0.5, *lig[:4], lig[4][:, :2], prec=1)
    check_search(got[0][:2], got[1][:2], r64, ridx,
                 lambda r: O.energy_map(grids, 0.5, lig[0][0], *lig[1:4], lig[4][0, r]))


def test_caller_owned_memory_and_graphs():
    import torch
    grids, lig = workload(64, 5, 20, 30)
    dev = [torch.from_numpy(a).cuda() for a in lig]
    with Receptor(grids, 0.5) as rec:
        want = rec.search(*lig)
        for count in (1, 4, 6, 30):
            q = dev[4][:, :count].contiguous()
            e = torch.empty(count, dtype=torch.float32, device="cuda")
            i = torch.empty(count, 3, dtype=torch.int32, device="cuda")
            L.check(L.lib().cdk_search_device_noalloc(
                rec.handle, lig[0].shape[1], 1, *(C.c_void_p(t.data_ptr()) for t in dev[:4]), count,
                C.c_void_p(q.data_ptr()), C.c_void_p(e.data_ptr()), C.c_void_p(i.data_ptr()), None))
            same((e.cpu().numpy(), i.cpu().numpy()), want, count)
    with Receptor(grids, 0.5, use_graphs=1) as rec:
        for count in (1, 1, 1, 8, 8, 8, 2, 2, 2):
            same(rec.search(*lig[:4], lig[4][:, :count]), want, count)


@pytest.mark.parametrize("n,box", [(32, 9), (64, 40)])
def test_infinite_receptor(n, box):
    """A receptor grid that holds an infinity: the same bits from both kernels (NaN energies among them)."""
    grids, lig = workload(n, 4, box, 40)
    grids[1, 2, 3, 4] = np.inf
    with Receptor(grids, 0.5) as rec:
        want = rec.search(*lig)
        for count in (1, 3):
            same(rec.search(*lig[:4], lig[4][:, :count]), want, count)
