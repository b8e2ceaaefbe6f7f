"""The decode-window plan where its way of placing pairs changes: 64 and 65 tokens (a token mask holds 64), tokens that name an
expert twice, experts without a blob, an expert table too large for masks.  Exact against the oracle."""
import numpy as np
import pytest
import torch

from basalt_b200 import moe
from oracle import oracle as O
from tests.test_experts_gpu import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,k,E", [(1, 1, 32), (1, 10, 512), (16, 10, 512), (63, 8, 96), (64, 10, 512), (64, 16, 1024), (65, 10, 512), (102, 10, 512), (64, 8, 2048)])
@pytest.mark.parametrize("ids_kind", ["distinct", "twice", "holes"])
def test_plan_places(lib, cuda, T, k, E, ids_kind):
    rng = np.random.default_rng(T * 131 + k + E)
    ids = np.stack([rng.permutation(E)[:k] for _ in range(T)]).astype(np.int32)
    if ids_kind == "twice" and k > 1:
        ids[T // 2, k - 1] = ids[T // 2, 0]
        ids[0, :2] = 3
    blobs = (rng.integers(1, 1 << 40, E) * 16).astype(np.uint64)
    if ids_kind == "holes":
        ids[rng.random(ids.shape) < 0.2] = -1
        blobs[rng.random(E) < 0.3] = 0
    ptr, start, ng, dst, tok = (t.cpu().numpy() for t in moe.moe_plan(dev(ids.reshape(-1)), k, E, dev(blobs.view(np.int64))))
    optr, ostart, ong, odst, otok = O.moe_plan(ids, k, E, blobs)
    g = int(ong)
    n = int(ostart[g])
    assert int(ng[0]) == g and np.array_equal(ptr[:g].view(np.uint64), optr[:g].view(np.uint64)) and np.array_equal(start[:g + 1], ostart[:g + 1])
    assert np.array_equal(dst[:n], odst[:n]) and np.array_equal(tok[:n], otok[:n])
    torch.cuda.synchronize()
