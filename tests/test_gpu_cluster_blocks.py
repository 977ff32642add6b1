"""The conformer selection's blocks of 32 candidates against the oracle: counts around the block
edges, centre limits met on the first, inside and past a block, and limits that never stop."""
import numpy as np
import pytest

from cdocker_b200 import synth
from cdocker_b200.conformers import cluster_conformers
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_conf", [1, 2, 31, 32, 33, 64, 65, 97, 1057])
@pytest.mark.parametrize("cutoff", [0.5, 1.5, 3.0])
def test_blocks_vs_oracle(n_conf, cutoff):
    x, e = synth.conformer_ensemble(n_conf, n_atoms=12, n_conf=n_conf, n_rotors=5)
    for limit in (1, 2, 3, 32, 33, 100, 0):
        got = cluster_conformers(x, e, cutoff, limit)
        np.testing.assert_array_equal(got, O.cluster_conformers(x, e, cutoff, limit))


def test_threads_and_sizes_share_nothing():
    """Calls of changing size (past the kept memory's bound too) from several threads at once."""
    from concurrent.futures import ThreadPoolExecutor
    sets = [synth.conformer_ensemble(s, n_atoms=a, n_conf=n, n_rotors=4)
            for s, a, n in ((1, 20, 300), (2, 9, 40), (3, 400, 4000), (4, 30, 500), (5, 6, 1))]
    want = [O.cluster_conformers(x[:600], e[:600], 1.5, 20) for x, e in sets]

    def one(i):
        x, e = sets[i % len(sets)]
        cluster_conformers(x, e, 1.5, 20)
        return cluster_conformers(x[:600], e[:600], 1.5, 20)

    with ThreadPoolExecutor(4) as ex:
        for i, got in enumerate(ex.map(one, range(20))):
            np.testing.assert_array_equal(got, want[i % len(sets)])
