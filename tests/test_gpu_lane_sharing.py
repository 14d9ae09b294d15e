"""Per-thread classes with several lanes per quartet (short lists and heavy bras)."""
import numpy as np
import pytest

from chronusq_public_b200.basis import BasisSet
from chronusq_public_b200.molecule import Molecule, single_water, water_cluster
from oracle import oracle as O

pytestmark = pytest.mark.gpu

TOL_G = 1e-10          # the parity bound of every FP64 build


def _density(n, seed, scale=1.0):
    a = np.random.default_rng(seed).uniform(-scale, scale, (n, n))
    return np.asfortranarray(0.5 * (a + a.T))


def _molecule(name):
    if name == "Ne":
        return Molecule(atoms=[10], coords=np.zeros((1, 3)))
    n = int(name)
    return single_water(7) if n == 1 else water_cluster(n, 7)


# from one atom (every list shorter than a warp: 32 lanes per quartet, more than most bras
# have primitive pairs) to lists that leave two lanes, then one lane for each quartet
@pytest.mark.parametrize("name,basis", [("Ne", "cc-pvtz"), ("1", "sto-3g"), ("1", "cc-pvdz"), ("2", "6-31g*"),
                                        ("3", "cc-pvdz"), ("5", "6-31g*"), ("6", "cc-pvdz")])
@pytest.mark.parametrize("uhf", [False, True])
def test_build_matches_oracle(name, basis, uhf):
    from chronusq_public_b200.aointegrals import AOIntegrals
    mol = _molecule(name)
    bs = BasisSet(basis, mol.atoms, mol.coords)
    ob = O.OracleBasis.from_basis(bs)
    Ps = _density(bs.nbasis, 1)
    Pz = _density(bs.nbasis, 2, 0.3) if uhf else None
    ints = AOIntegrals(bs)
    got = ints.formPT(Ps, Pz)
    ref = O.form_pt(ob, Ps, Pz)
    assert ints.stats()["quartets"] == ref[2]
    for g, r in zip(got, ref[:2]):
        if r is not None:
            assert np.abs(g - r).max() <= TOL_G
    ints.close()
