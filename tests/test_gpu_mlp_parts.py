"""The gradient of a layer's input in the guess network: which parts of its sum are formed apart,
and the passes of large batches (128 x 128 tiles)."""
import numpy as np
import pytest

from test_gpu_mlp_passes import _gpu, test_backward_pass as check_backward_pass

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("batch", [1, 63, 200, 700, 2048, 2500, 20000])
def test_parts_of_the_input_gradient(batch):
    """256 products 2^40, -2^40 and ones, laid out so that a sum in parts of 64 or more is exactly
    208 in any order of the parts, and a sum in shorter ones is not: +2^40 and -2^40 would stand
    in different parts, with ones after the second that its part loses."""
    _gpu()
    from chronusq_public_b200.guess_model import NFEAT, PairMLP
    m = PairMLP(width=256, layers=1, seed=3, maxf=16)
    m.set_weights([np.zeros((256, NFEAT)), np.ones((256, 256))], [np.zeros(256), np.zeros(256)])
    row = np.ones(256)
    row[:16] = row[32:48] = 0.0
    row[0], row[32] = 2.0**40, -2.0**40
    _, cache = m.forward(torch.ones((batch, NFEAT), dtype=torch.bfloat16, device="cuda"), keep=True)
    dout = torch.tensor(np.tile(row, (batch, 1)), dtype=torch.float32, device="cuda")
    gW, gb = m.backward(dout, cache)
    # SiLU'(0) = 1/2; the sums over the rows are whole numbers below 2^24
    assert torch.equal(gb[0], torch.full((256,), 104.0 * batch, device="cuda"))
    assert torch.equal(gW[0], torch.full((256, NFEAT), 104.0 * batch, device="cuda"))


@pytest.mark.parametrize("batch", [2500, 20000])   # no split, 64 x 64 and 128 x 128 tiles
def test_backward_of_large_batches(batch):
    check_backward_pass(batch, 256)


def test_backward_of_layers_of_both_tile_sizes():
    """A weight gradient of large tiles (2304 x 2304) after one of small tiles."""
    _gpu()
    from chronusq_public_b200.guess_model import NFEAT, PairMLP
    m = PairMLP(width=2304, layers=2, seed=3, maxf=12)
    rng = np.random.default_rng(4)
    X = torch.tensor(rng.standard_normal((70, NFEAT)), dtype=torch.float32, device="cuda").to(torch.bfloat16)
    out, cache = m.forward(X, keep=True)
    dout = torch.tensor(rng.standard_normal(out.shape), dtype=torch.float32, device="cuda")
    gW, gb = m.backward(dout, cache)
    d, tol = dout.to(torch.bfloat16).double(), 0.0
    eps = (70 + 2) * 2.0**-23
    for i in (2, 1, 0):
        h, z = cache[i][0].double(), cache[i][1].double()
        if i < 2:
            W = m.Wbf[i + 1].double()
            s = torch.sigmoid(z)
            g = s * (1.0 + z * (1.0 - s))
            # one BF16 rounding here and those of the layers above, FP32 sums and SiLU' (|SiLU'| < 1.1)
            tol = 2.0**-8 * ((d @ W) * g).abs() + 1e-5 * (d.abs() @ W.abs()) + 1.1 * (tol @ W.abs() if i == 0 else 0.0)
            d = (d @ W) * g
        extra = tol.t() @ h.abs() if i < 2 else 0.0
        assert bool(((gW[i].double() - d.t() @ h).abs() <= extra + eps * (d.abs().t() @ h.abs()) + 1e-30).all())
        extra = tol.sum(0) if i < 2 else 0.0
        assert bool(((gb[i].double() - d.sum(0)).abs() <= extra + eps * d.abs().sum(0) + 1e-30).all())
