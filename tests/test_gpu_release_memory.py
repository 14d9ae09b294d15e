"""The memory that closed contexts leave for later ones can be given back."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def test_release_memory():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from chronusq_public_b200 import _lib
    from test_gpu_pool import _fock
    first = _fock(3)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    n = _lib.release_memory()
    assert 0 < n <= 256 << 20
    # the driver hands memory out in pages of 2 MiB, several small blocks to a page
    assert torch.cuda.mem_get_info()[0] - before >= n // 2
    assert _lib.release_memory() == 0
    torch.testing.assert_close(_fock(3), first, rtol=0, atol=1e3 * 2.0**-53 * float(first.abs().max()))
    with pytest.raises(_lib.CqgError):
        _lib.release_memory(-1)


def test_buffers_of_a_context_closed_inside_a_capture():
    """The wait for the device fails there, so nothing of the context may be handed to another one."""
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from chronusq_public_b200 import _lib
    from chronusq_public_b200.aointegrals import AOIntegrals
    from chronusq_public_b200.basis import BasisSet
    from chronusq_public_b200.molecule import water_cluster
    from test_gpu_pool import _fock
    first = _fock(2)
    mol = water_cluster(2, seed=5)
    ints = AOIntegrals(BasisSet("6-31g*", mol.atoms, mol.coords))
    _lib.release_memory()
    torch.cuda.synchronize()
    with pytest.raises(RuntimeError):   # the wait also ends the capture
        with torch.cuda.graph(torch.cuda.CUDAGraph()):
            ints.close()
    torch.cuda.synchronize()
    assert _lib.release_memory() == 0
    torch.testing.assert_close(_fock(2), first, rtol=0, atol=1e3 * 2.0**-53 * float(first.abs().max()))
