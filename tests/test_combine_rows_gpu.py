"""The combine at numbers of rows around those it requests at once (12), with and without the shared and residual rows, widths that do not
fill a block: against 64 bits (bound: (k + 2) roundings of 2^-24 of the sum of magnitudes) and bit for bit against the same rows named by slots."""
import numpy as np
import pytest
import torch

from basalt_b200 import moe

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 11, 12, 13, 25])
@pytest.mark.parametrize("T,H", [(1, 4), (3, 516), (9, 2048)])
def test_combine_rows(lib, cuda, k, T, H):
    rng = np.random.default_rng(k * H)
    rows = rng.standard_normal((T * k, H)).astype(np.float32)
    w = rng.random((T, k)).astype(np.float32)
    sh = rng.standard_normal((T, H)).astype(np.float32)
    dev = lambda a: torch.from_numpy(a).cuda()
    slot = dev(np.arange(T * k, dtype=np.int32).reshape(T, k))
    for shared in (None, dev(sh)):
        y = moe.moe_combine(dev(rows), None, dev(w), shared=shared)
        ys = moe.moe_combine(dev(rows), slot, dev(w), shared=shared)
        assert torch.equal(y.view(torch.int32), ys.view(torch.int32))
        terms = rows.reshape(T, k, H).astype(np.float64) * w[:, :, None]
        want, mag = terms.sum(1), np.abs(terms).sum(1)
        if shared is not None:
            want, mag = want + sh, mag + np.abs(sh)
        assert (np.abs(y.cpu().numpy() - want) <= (k + 2) * 2.0**-24 * mag).all()
