"""The autotuner's candidates: the default launch of a list is one of them."""
import numpy as np
import pytest

from chronusq_public_b200.basis import BasisSet
from chronusq_public_b200.molecule import water_cluster
from test_gpu_parity import TOL_G, _aoi, rand_sym

pytestmark = pytest.mark.gpu


def test_default_launch_is_a_candidate_and_is_kept():
    """Lists this short take the same few microseconds in every shape, so some keep the default
    claim (0), with the resident grid that was timed written out."""
    mol = water_cluster(3, 12)
    bs = BasisSet("cc-pvdz", mol.atoms, mol.coords)
    D = rand_sym(bs.nbasis, 53)
    ints = _aoi()(bs)
    before = ints.schedule()
    G0, _ = ints.formPT(D)
    ints.autotune_next()
    G1, _ = ints.formPT(D)
    after = ints.schedule()
    tuned = [k for k, c in enumerate(after["cta_per_sm"]) if c > 0]
    assert set(before["cta_per_sm"]) == {0} and tuned
    assert any(after["quartets_per_warp"][k] == 0 for k in tuned)
    G2, _ = ints.formPT(D)
    assert np.abs(G1 - G0).max() <= TOL_G and np.abs(G2 - G0).max() <= TOL_G
    ints.close()
