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
