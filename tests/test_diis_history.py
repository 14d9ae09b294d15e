"""The DIIS rings against sums over plain lists of matrices, past their size and with the oldest dropped."""
import types

import numpy as np
import pytest

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("size,nmat,nerr,count", [(1, 2, 1, 3), (4, 2, 1, 3), (4, 4, 2, 4), (4, 4, 2, 11)])
def test_history(size, nmat, nerr, count):
    from chronusq_public_b200.scf import _DIISHistory
    h = _DIISHistory(types.SimpleNamespace(torch=torch, nDIISExtrap=size, maxSCFIter=50))
    g = torch.Generator().manual_seed(count)
    draw = lambda k: [torch.randn(5, 5, dtype=torch.float64, generator=g) for _ in range(k)]
    for _ in range(2):   # cleared, it starts again
        mats, errs = [], []
        for _ in range(count):
            mats.append(draw(nmat))
            errs.append(draw(nerr))
            norm = h.append(mats[-1], errs[-1])
            assert norm == pytest.approx(max(float(torch.linalg.norm(e)) for e in errs[-1]), rel=1e-14)
            mats, errs = mats[-size:], errs[-size:]
        m = len(errs)
        assert len(h) == m
        ref = [[sum(float((a * b).sum()) for a, b in zip(x, y)) for y in errs] for x in errs]
        np.testing.assert_allclose(h.gram(), ref, rtol=0, atol=50 * 2.0**-52 * max(map(max, ref)))
        for n in {m, max(1, m - 1)}:
            c = [0.7, -1.5, 2.25, 0.125][:n]
            ext = h.extrapolate(c)
            for j in range(nmat):
                want = sum(x * q[j] for x, q in zip(c, mats[m - n:]))
                torch.testing.assert_close(ext[j], want, rtol=0, atol=8 * 2.0**-52 * 20)
        h.clear()
