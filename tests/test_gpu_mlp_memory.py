"""Device memory of a prediction: the hidden layers share buffers when no backward pass follows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("layers", [1, 2, 4])
def test_forward_without_backward(layers):
    from test_gpu_mlp_passes import _gpu
    _gpu()
    from chronusq_public_b200.guess_model import NFEAT, PairMLP
    m, rows = PairMLP(width=256, layers=layers, seed=3, maxf=14), 100_000
    X = torch.tensor(np.random.default_rng(1).standard_normal((rows, NFEAT)), dtype=torch.float32,
                     device="cuda").to(torch.bfloat16)
    kept, cache = m.forward(X, keep=True)
    assert len(cache) == layers + 1
    del cache
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    base = torch.cuda.memory_allocated()
    out, cache = m.forward(X)
    assert cache == [] and torch.equal(out, kept)
    # per row: the output, one FP32 and at most two BF16 hidden layers; blocks are rounded up to 2 MiB
    per_row = 4 * 14 * 14 + 256 * (4 + 2 * min(layers, 2))
    assert torch.cuda.max_memory_allocated() - base <= rows * per_row + 3 * (2 << 20)
