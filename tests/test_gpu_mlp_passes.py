"""Whole passes of the guess network and the edges of its matrix products: tile remainders, rows
that 16-byte copies cannot take, partial sums in and across blocks."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _gpu():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")


@pytest.mark.parametrize("form", ["nt", "tn", "nn"])
@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (63, 65, 31), (64, 64, 33), (65, 72, 160), (200, 196, 57), (130, 40, 1030),
                                   (2500, 2304, 40)])
def test_product_edges(M, N, K, form):
    _gpu()
    from chronusq_public_b200 import _lib
    L = _lib.lib()
    rng = np.random.default_rng(M + N + K)
    A, B = (torch.tensor(rng.standard_normal(s), dtype=torch.bfloat16, device="cuda") for s in ((M, K), (N, K)))
    C = torch.ones((M, N), device="cuda")
    a, sa = (A.t().contiguous(), (1, M)) if form == "tn" else (A, (K, 1))
    b, sb = (B, (K, 1)) if form == "nt" else (B.t().contiguous(), (1, N))
    p = lambda x: ctypes.c_void_p(x.data_ptr())
    _lib.check(L.cqg_mlp_gemm_bf16(p(a), *sa, p(b), *sb, p(C), N, M, N, K, None, None, 0, 0, 1, None))
    torch.cuda.synchronize()
    ref = 1.0 + A.double() @ B.double().t()
    # products of two BF16 are exact in FP32; K + 2 roundings of partial sums
    tol = (K + 2) * 2.0**-23 * (1.0 + A.double().abs() @ B.double().abs().t())
    assert bool(((C.double() - ref).abs() <= tol).all())


@pytest.mark.parametrize("batch,width", [(1, 256), (65, 256), (2048, 256), (301, 20), (64, 33)])
def test_backward_pass(batch, width):
    _gpu()
    from chronusq_public_b200.guess_model import NFEAT, PairMLP
    m = PairMLP(width=width, layers=1, seed=3, maxf=14)
    rng = np.random.default_rng(batch)
    X = torch.tensor(rng.standard_normal((batch, NFEAT)), dtype=torch.float32, device="cuda").to(torch.bfloat16)
    out, cache = m.forward(X, keep=True)
    dout = torch.tensor(rng.standard_normal(out.shape), dtype=torch.float32, device="cuda")
    gW, gb = m.backward(dout, cache)
    (x, z), (h, _) = ((a.double(), b.double()) for a, b in cache)
    d1 = dout.to(torch.bfloat16).double()
    W1 = m.Wbf[1].double()
    s = torch.sigmoid(z)
    d0 = (d1 @ W1) * (s * (1.0 + z * (1.0 - s)))
    # dZ of the hidden layer: one BF16 rounding on either side, FP32 sums and SiLU' (|SiLU'| < 1.1)
    t0 = 2.0**-8 * d0.abs() + 1e-5 * (d1.abs() @ W1.abs())
    eps = (batch + 2) * 2.0**-23
    for got, ref, tol in ((gW[1], d1.t() @ h, eps * (d1.abs().t() @ h.abs())),
                          (gb[1], d1.sum(0), eps * d1.abs().sum(0)),
                          (gW[0], d0.t() @ x, t0.t() @ x.abs() + eps * (d0.abs().t() @ x.abs())),
                          (gb[0], d0.sum(0), t0.sum(0) + eps * d0.abs().sum(0))):
        assert got.shape == ref.shape
        assert bool(((got.double() - ref).abs() <= tol + 1e-30).all())


@pytest.mark.parametrize("layers", [2, 9])   # fewer tensors than a launch takes, and more
def test_adam_of_all_tensors(layers):
    _gpu()
    from chronusq_public_b200.guess_model import PairMLP
    m = PairMLP(width=40, layers=layers, seed=5, maxf=14)
    rng = np.random.default_rng(7)
    gW, gb = ([torch.tensor(rng.standard_normal(x.shape), dtype=torch.float32, device="cuda") for x in xs]
              for xs in (m.W, m.b))
    before = [x.double().clone() for x in m.W + m.b]
    m.adam(gW, gb, 1e-3, 0.01)
    for k, (x, x0, g) in enumerate(zip(m.W + m.b, before, gW + gb)):
        g = g.double() + (0.01 if k < len(m.W) else 0.0) * x0
        ref = x0 - 1e-3 * g / (g.abs() + 1e-8)   # the first step: both moments are corrected to g and g^2
        # a step of 1e-3 to a few parts in 1e5 (its corrections cancel 24-bit numbers), and the sum's rounding
        assert bool(((x.double() - ref).abs() <= 1e-3 * 1e-4 + 2.0**-23 * ref.abs()).all())
    assert all(torch.equal(b, w.to(torch.bfloat16)) for b, w in zip(m.Wbf, m.W))
