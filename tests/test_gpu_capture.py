"""Dipole matrices captured in a CUDA graph by a context that holds no side streams yet."""
import ctypes

import numpy as np
import pytest

from chronusq_public_b200.basis import BasisSet
from chronusq_public_b200.molecule import water_cluster
from test_gpu_parity import _aoi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("timed_setup", [True, False])
def test_dipole_in_a_graph(timed_setup):
    import torch
    from chronusq_public_b200 import _lib
    mol = water_cluster(2, 3)
    bs = BasisSet("6-31g*", mol.atoms, mol.coords)
    # as many contexts as the library keeps stream sets for, and one more: none is left to lease
    held = [_aoi()(bs) for _ in range(9)]
    ref = held[0].computeDipole()
    L = _lib.lib()
    ctx = ctypes.c_void_p()
    _lib.check(L.cqg_create(ctypes.byref(ctx), 0))
    _lib.check(L.cqg_set_timing(ctx, int(timed_setup)), ctx)   # a timed context takes no side streams
    flat = [np.ascontiguousarray(x) for x in bs.flat()]
    ptr = [x.ctypes.data_as(ctypes.POINTER(ctypes.c_int if x.dtype.kind == "i" else ctypes.c_double)) for x in flat]
    _lib.check(L.cqg_set_basis(ctx, len(flat[0]), *ptr), ctx)
    _lib.check(L.cqg_set_timing(ctx, 0), ctx)
    n = bs.nbasis
    D = torch.zeros((3, n, n), dtype=torch.float64, device="cuda")
    O = np.zeros(3)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        _lib.check(L.cqg_dipole(ctx, O.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), ctypes.c_void_p(D.data_ptr()),
                                n, 1, st), ctx)
    g.replay()
    torch.cuda.synchronize()
    # the same kernels on the same numbers
    assert np.abs(D.cpu().numpy() - ref).max() <= 1e-14
    del g
    L.cqg_destroy(ctx)
    for h in held:
        h.close()
