"""One-electron class kernels against the CPU oracle: few and many charges, every pair class."""
import numpy as np
import pytest

from chronusq_public_b200.basis import BasisSet
from chronusq_public_b200.molecule import single_water, water_cluster
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# absolute; V sums up to 300 charges of at most unit size besides the nuclei
TOL = {"S": 1e-12, "T": 1e-11, "V": 1e-10, "D": 1e-11}


# no charge, fewer and more than the lanes of a warp, and a remainder of one
@pytest.mark.parametrize("ncharge", [0, 1, 7, 33, 300])
@pytest.mark.parametrize("nwater,basis", [(1, "cc-pvtz"), (3, "cc-pvdz")])
def test_one_electron_matrices_match_oracle(nwater, basis, ncharge):
    from chronusq_public_b200.aointegrals import AOIntegrals
    mol = single_water(5) if nwater == 1 else water_cluster(nwater, 5)
    bs = BasisSet(basis, mol.atoms, mol.coords)
    rng = np.random.default_rng(ncharge)
    Z = rng.uniform(-1.0, 1.0, ncharge)
    R = rng.uniform(-6.0, 6.0, (ncharge, 3))
    if ncharge > 1:
        R[0] = mol.coords[0]           # a charge on a nucleus: T = 0 for the pairs of that atom
    ob = O.OracleBasis.from_basis(bs)
    ref = dict(zip("STV", O.one_e(ob, Z, R)))
    ints = AOIntegrals(bs)
    got = dict(zip("STV", ints.computeAOOneE(Z, R)))
    got["D"], ref["D"] = ints.computeDipole(), np.stack(O.dipole(ob))
    for k in got:
        assert np.abs(got[k] - ref[k]).max() <= TOL[k], k
    for M in (got["S"], got["T"], got["V"]):
        assert np.array_equal(M, M.T)
    ints.close()
