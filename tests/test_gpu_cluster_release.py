"""The device memory kept by the conformer selection is given back on request, and with a context."""
import numpy as np
import pytest

from cdocker_b200 import Receptor, synth
from cdocker_b200.conformers import cluster_conformers, release_workspaces

pytestmark = pytest.mark.gpu


def test_kept_memory_is_given_back():
    x, e = synth.conformer_ensemble(5, n_atoms=20, n_conf=150, n_rotors=4)
    want = cluster_conformers(x, e, 1.5, 40)
    assert release_workspaces() >= 1 and release_workspaces() == 0
    assert np.array_equal(cluster_conformers(x, e, 1.5, 40), want)
    Receptor(np.zeros((2, 32, 32, 32), np.float32), 0.5).close()
    assert release_workspaces() == 0
    assert np.array_equal(cluster_conformers(x, e, 1.5, 40), want)
    assert release_workspaces() == 1
