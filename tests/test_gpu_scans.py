"""Offsets of the screening's tasks by the single-block scan and by the device-wide one: a batch of
copies of one molecule has copies of its lists, whichever scan it is large enough for."""
import numpy as np
import pytest

from chronusq_public_b200.basis import BasisSet
from chronusq_public_b200.molecule import single_water
from oracle import oracle as O
from test_gpu_parity import TOL_G, rand_sym

pytestmark = pytest.mark.gpu

# tasks of one water in 6-31G(d): the bra pairs of every class block; the single-block scan takes
# four offsets a task, 32768 in all
LIMIT = 8192


def _tasks(bs):
    ls = [s.l for s in bs.shells]
    pairs = {}
    for i, a in enumerate(ls):
        for b in ls[:i + 1]:
            c = (max(a, b), min(a, b))
            pairs[c] = pairs.get(c, 0) + 1
    order = sorted(pairs)
    return sum(pairs[b] * (order.index(b) + 1) for b in order)


@pytest.mark.parametrize("fraction", [0.1, 1.0, 1.02, 2.5])
def test_copies_of_one_molecule(fraction):
    from chronusq_public_b200.batch import BatchAOIntegrals
    mol = single_water(2)
    bs = BasisSet("6-31g*", mol.atoms, mol.coords)
    copies = int(fraction * LIMIT / _tasks(bs))
    assert (copies * _tasks(bs) <= LIMIT) == (fraction <= 1.0)
    D = rand_sym(bs.nbasis, 5)
    ref, _, nq = O.form_pt(O.OracleBasis.from_basis(bs), D, thresh=1e-12)
    B = BatchAOIntegrals([bs] * copies, thresholdSchwartz=1e-12)
    PT = B.formPT(B.pack([D] * copies))
    assert B.stats()["quartets"] == copies * nq
    for m in range(copies):
        assert np.abs(B.view(PT, m).cpu().numpy() - ref).max() <= TOL_G
    B.close()
