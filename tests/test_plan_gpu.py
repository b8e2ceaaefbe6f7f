"""The decode-window plan where its way of placing pairs changes: 64 and 65 tokens (a token mask holds 64), tokens that name an
expert twice, experts without a blob, an expert table too large for masks, and tables that fill the kernels' shared memory to its
last bytes.  Exact against the oracle."""
import numpy as np
import pytest
import torch

from basalt_b200 import capi, moe
from oracle import oracle as O
from tests.test_experts_gpu import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,k,E", [(1, 1, 32), (1, 10, 512), (16, 10, 512), (63, 8, 96), (64, 10, 512), (64, 16, 1024), (65, 10, 512), (102, 10, 512), (64, 8, 2048),
                                   (1, 8, 2040), (16, 8, 2016), (40, 8, 1984), (56, 13, 1920), (64, 4, 2000), (64, 8, 1952), (64, 8, 1960)])
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


@pytest.mark.parametrize("T,k,E", [(1, 8, 1024), (1016, 8, 1024), (1020, 8, 1024), (1024, 8, 1024), (512, 8, 2048)])
def test_gathered_plan_fills_its_tables(lib, cuda, T, k, E):
    """bsx_ep_plan up to its documented limits; the order of the entries inside a group is not fixed."""
    rng = np.random.default_rng(T + E)
    ids = np.stack([rng.permutation(E)[:k] for _ in range(T)]).astype(np.int32)
    blobs = (rng.integers(1, 1 << 40, E) * 16).astype(np.uint64)
    blobs[rng.random(E) < 0.3] = 0
    n = T * k
    lb = capi.lib()
    i32 = dict(dtype=torch.int32, device="cuda")
    idd, table = dev(ids.reshape(-1)), dev(blobs.view(np.int64))
    ptr, start, ng = torch.zeros(E + 3, dtype=torch.int64, device="cuda"), torch.zeros(E + 3, **i32), torch.zeros(1, **i32)
    dst, tok = torch.zeros(n, **i32), torch.zeros(n, **i32)
    capi.check("bsx_ep_plan", lb.bsx_ep_plan(idd.data_ptr(), n, k, 0, 0, E, table.data_ptr(), 0, 0, 0, None, ptr.data_ptr(), start.data_ptr(), ng.data_ptr(),
                                             dst.data_ptr(), tok.data_ptr(), moe._stream(None)))
    torch.cuda.synchronize()
    optr, ostart, og, odst, _ = O.moe_plan(ids, k, E, blobs)
    m = int(ostart[og])
    start, dst, tok = start.cpu().numpy(), dst.cpu().numpy(), tok.cpu().numpy()
    assert int(ng.item()) == og and np.array_equal(ptr.cpu().numpy()[:og].view(np.uint64), optr[:og]) and np.array_equal(start[:og + 1], ostart[:og + 1])
    for g in range(og):
        assert np.array_equal(np.sort(dst[start[g]:start[g + 1]]), np.sort(odst[ostart[g]:ostart[g + 1]]))
    assert np.array_equal(tok[:m], dst[:m] // k)


def test_gathered_plan_refuses_larger_tables(lib, cuda):
    one = torch.zeros(1, dtype=torch.int64, device="cuda").data_ptr()
    for n, E in ((8193, 32), (8192, 1056), (4097, 2048)):
        assert capi.lib().bsx_ep_plan(one, n, 8, 0, 0, E, one, 0, 0, 0, None, one, one, one, one, one, moe._stream(None)) == capi.E_LIMIT
