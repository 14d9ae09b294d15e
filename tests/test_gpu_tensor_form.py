"""The tensor-core form of the classes that also have a per-thread form, on bases without d shells:
(pp|pp) has both, and its expansion tables are those of the basis in use."""
import ctypes

import numpy as np
import pytest

from chronusq_public_b200.basis import BasisSet
from chronusq_public_b200.molecule import single_water, water_cluster
from oracle import oracle as O
from test_gpu_parity import TOL_G, _aoi, rand_sym

pytestmark = pytest.mark.gpu

SP = ["sto-3g", "6-31g"]
PP = "(pp|pp)"


def _check(ints, bs, D):
    G, _ = ints.formPT(D)
    st = ints.stats()
    Gr, _, nr = O.form_pt(O.OracleBasis.from_basis(bs), D)
    assert st["quartets"] == nr
    assert np.abs(G - Gr).max() <= TOL_G


@pytest.mark.parametrize("basis", SP)
@pytest.mark.parametrize("how", ["forced", "autotuned"])
def test_sp_basis(basis, how):
    mol = water_cluster(3, 11)
    bs = BasisSet(basis, mol.atoms, mol.coords)
    ints = _aoi()(bs)
    if how == "forced":
        ints.setSchedule(cta_per_sm=8, warps_per_cta=2, quartets_per_warp=4, warp_form=1)
        from chronusq_public_b200 import _lib
        assert ints.schedule()["warp_form"][_lib.class_names().index(PP)] == 1
    else:
        ints.autotune_next()
    for seed in (41, 42):
        _check(ints, bs, rand_sym(bs.nbasis, seed))
    ints.close()


def test_s_only_basis():
    """No class of the basis has a tensor form: a forced one changes nothing."""
    from chronusq_public_b200.molecule import Molecule
    mol = Molecule([1, 1], np.array([[0.0, 0.0, 0.0], [0.0, 0.0, 1.4]]))
    bs = BasisSet("6-31g", mol.atoms, mol.coords)
    ints = _aoi()(bs)
    ints.setSchedule(warp_form=1)
    _check(ints, bs, rand_sym(bs.nbasis, 7))
    ints.autotune_next()
    _check(ints, bs, rand_sym(bs.nbasis, 8))
    ints.close()


@pytest.mark.parametrize("basis", SP)
@pytest.mark.parametrize("how", ["forced", "autotuned"])
def test_sp_batch(basis, how):
    from chronusq_public_b200.batch import BatchAOIntegrals
    mols = [single_water(2), water_cluster(2, 3), water_cluster(3, 4)]
    bss = [BasisSet(basis, m.atoms, m.coords) for m in mols]
    B = BatchAOIntegrals(bss, thresholdSchwartz=1e-12)
    if how == "forced":
        _force(B)
    else:
        B.autotune_next()
    for seed in (5, 6):
        Ds = [rand_sym(bs.nbasis, seed + 10 * i) for i, bs in enumerate(bss)]
        G = B.formPT(B.pack(Ds))
        for m, (bs, D) in enumerate(zip(bss, Ds)):
            Gr, _, _ = O.form_pt(O.OracleBasis.from_basis(bs), D, thresh=1e-12)
            assert np.abs(B.view(G, m).cpu().numpy() - Gr).max() <= TOL_G
    B.close()


def _force(ints):
    from chronusq_public_b200 import _lib
    n = int(ints._L.cqg_schedule_lists())
    arr = lambda v: (ctypes.c_int * n)(*[v] * n)
    _lib.check(ints._L.cqg_set_schedule(ints._ctx, arr(8), arr(2), arr(4), arr(1)), ints._ctx)


@pytest.mark.parametrize("how", ["forced", "autotuned"])
def test_new_basis_on_one_context(how):
    """d shells first, then an s and p basis of more pairs, then d shells again: each with the
    tensor form that the first one was left with."""
    from chronusq_public_b200 import _lib
    first = water_cluster(2, 3)
    big = water_cluster(5, 4)
    a, b = BasisSet("cc-pvdz", first.atoms, first.coords), BasisSet("6-31g", big.atoms, big.coords)
    ints = _aoi()(a)
    if how == "forced":
        _force(ints)
    else:
        ints.autotune_next()
    _check(ints, a, rand_sym(a.nbasis, 9))
    if how == "autotuned":   # whatever the tuner chose, the form with tables is what is tested
        _force(ints)
    for bs in (b, a):
        flat = [np.ascontiguousarray(x) for x in bs.flat()]
        ptr = [x.ctypes.data_as(ctypes.POINTER(ctypes.c_int if x.dtype.kind == "i" else ctypes.c_double)) for x in flat]
        _lib.check(ints._L.cqg_set_basis(ints._ctx, len(flat[0]), *ptr), ints._ctx)
        ints.nBasis, ints.basisSet = bs.nbasis, bs
        _check(ints, bs, rand_sym(bs.nbasis, 10))
    ints.close()
