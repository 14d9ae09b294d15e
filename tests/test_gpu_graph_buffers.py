"""A captured contraction keeps its buffers when a host-pointer call in graph mode needs larger ones."""
import numpy as np
import pytest

from chronusq_public_b200.basis import BasisSet
from chronusq_public_b200.molecule import single_water, water_cluster
from oracle import oracle as O
from test_gpu_parity import TOL_G, _aoi, rand_sym

pytestmark = pytest.mark.gpu


def test_replay_after_a_host_call_that_outgrew_the_buffers():
    import torch
    from chronusq_public_b200 import _lib
    mol, big = single_water(4), water_cluster(3, 12)
    bs, bs2 = (BasisSet("6-31g*", m.atoms, m.coords) for m in (mol, big))
    ob = O.OracleBasis.from_basis(bs)
    Ps, Pz = rand_sym(bs.nbasis, 5), rand_sym(bs.nbasis, 6, 0.2)
    ints = _aoi()(bs)
    P = torch.tensor(Ps, device="cuda")
    ints.formPT(P)
    nq = ints.stats()["quartets"]
    _lib.check(ints._L.cqg_set_graph_mode(ints._ctx, nq + 64, 1), ints._ctx)
    PT, _ = ints.formPT(P)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        ints.formPT(P, PTs=PT)
    a, b, _ = O.form_pt(ob, Ps, Pz)
    # two groups instead of one: larger accumulators and copies of X
    Ha, Hb = ints.formPT(Ps, Pz)
    assert np.abs(Ha - a).max() <= TOL_G and np.abs(Hb - b).max() <= TOL_G
    # another context may now hold any block that went back to the pool
    other = _aoi()(bs2)
    D2 = torch.tensor(rand_sym(bs2.nbasis, 8), device="cuda")
    G2, _ = other.formPT(D2)
    ref2 = G2.clone()
    ref, _, _ = O.form_pt(ob, Ps)
    for _ in range(2):
        PT.fill_(7.0)
        g.replay()
        torch.cuda.synchronize()
        assert np.abs(PT.cpu().numpy() - ref).max() <= TOL_G
        G2, _ = other.formPT(D2)
        assert float((G2 - ref2).abs().max()) <= TOL_G
    del g
    _lib.check(ints._L.cqg_set_graph_mode(ints._ctx, 0, 1), ints._ctx)
    Ha, Hb = ints.formPT(Ps, Pz)
    assert np.abs(Ha - a).max() <= TOL_G and np.abs(Hb - b).max() <= TOL_G
    other.close()
    ints.close()
