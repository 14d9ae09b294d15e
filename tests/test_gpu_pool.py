"""Contexts that fill the device pool past its limit, so that freed blocks replace older ones,
and a context made again from what it then holds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _fock(n):
    from chronusq_public_b200.aointegrals import AOIntegrals
    from chronusq_public_b200.basis import BasisSet
    from chronusq_public_b200.molecule import water_cluster
    mol = water_cluster(n, seed=3)
    bs = BasisSet("6-31g*", mol.atoms, mol.coords)
    ints = AOIntegrals(bs)
    D = np.random.default_rng(n).standard_normal((bs.nbasis, bs.nbasis))
    D = torch.tensor((D + D.T) * np.exp(-0.5 * np.abs(np.subtract.outer(*2 * [np.arange(bs.nbasis)]))), device="cuda")
    G = ints.formPT(D)[0].clone()
    ints.close()
    return G


@pytest.mark.parametrize("sizes", [(2, 12, 20, 28, 2), (2, 24, 3, 16, 2)])
def test_pool_past_its_limit(sizes):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    first = _fock(sizes[0])
    for n in sizes[1:-1]:
        assert bool(torch.isfinite(_fock(n)).all())
    # the same contraction up to the order of its FP64 atomics: about 1e3 terms an element
    torch.testing.assert_close(_fock(sizes[-1]), first, rtol=0, atol=1e3 * 2.0**-53 * float(first.abs().max()))
