"""Q6_K experts on the integer tensor-core stream where its launch changes: a few entries (the columns of a row split over two, four or
eight warps), many groups (whole rows), odd and even numbers of 256-column blocks a part, rows that do not fill the last block of
warps.  Bound 4e-4: four times the error of two int8 terms a row (1e-4)."""
import numpy as np
import pytest

from basalt_b200 import moe
from oracle import oracle as O
from tests.helpers import make_expert_blobs, rel_l2, stack_blobs
from tests.test_experts_gpu import dev, run_grouped

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,I", [(512, 512), (2048, 512), (1536, 1024), (3072, 512), (512, 2560)])
@pytest.mark.parametrize("groups", [[[3]], [[4], list(range(13)), [0, 7]], [[i % 13] for i in range(60)]], ids=["one", "three", "sixty"])
def test_q6k_rows(lib, cuda, H, I, groups):
    rng = np.random.default_rng(H + I)
    Lo, blobs = make_expert_blobs(rng, 3, O.T_Q6_K, O.T_Q6_K, H, I)
    L = moe.native_expert_layout(O.T_Q6_K, O.T_Q6_K, H, I)
    xd = dev(rng.standard_normal((13, H)).astype(np.float32))
    x = xd.cpu().numpy()
    ids = [i % 3 for i in range(len(groups))]
    n = sum(len(g) for g in groups)
    out = run_grouped(L, dev(stack_blobs(blobs)), ids, groups, xd, n).cpu().numpy()
    at = 0
    for e, toks in zip(ids, groups):
        want = O.expert_forward(Lo, blobs[e], x[toks], dtype=np.float64)
        assert rel_l2(out[at:at + len(toks)], want) < 4e-4, (e, rel_l2(out[at:at + len(toks)], want))
        at += len(toks)


@pytest.mark.parametrize("H,I", [(8704, 512), (512, 8704)])
def test_rows_beyond_the_integer_kernel_keep_their_24_bits(lib, cuda, H, I):
    """Bound 1e-5: fp32 sums of exactly decoded weights."""
    rng = np.random.default_rng(H)
    Lo, blobs = make_expert_blobs(rng, 1, O.T_Q6_K, O.T_Q6_K, H, I)
    L = moe.native_expert_layout(O.T_Q6_K, O.T_Q6_K, H, I)
    x = rng.standard_normal((3, H)).astype(np.float32)
    out = run_grouped(L, dev(stack_blobs(blobs)), [0], [[0, 1, 2]], dev(x), 3).cpu().numpy()
    assert rel_l2(out, O.expert_forward(Lo, blobs[0], x, dtype=np.float64)) < 1e-5


@pytest.mark.parametrize("t,H,I", [(O.T_Q6_K, 512, 512), (O.T_Q6_K, 1536, 1024), (O.T_Q6_K, 5632, 1024), (O.T_Q6_K, 7168, 512), (O.T_Q6_K, 512, 8192),
                                   (O.T_IQ1_M, 2048, 512), (O.T_IQ1_M, 7168, 512), (O.T_IQ1_M, 512, 5120)])
@pytest.mark.parametrize("sizes", [[41], [1, 4, 5, 8, 9], [3] * 33], ids=["deep", "ragged", "many"])
def test_column_blocks_and_runs(lib, cuda, t, H, I, sizes):
    """One, two and four column blocks a pass, full and ragged; one or two blocks an SM; rows split over warps or not; runs of row blocks
    that end inside a pass, and row blocks that the rows do not fill (512 over the three tiles of twelve warps)."""
    rng = np.random.default_rng(H + I + len(sizes))
    Lo, blobs = make_expert_blobs(rng, 2, t, t, H, I)
    L = moe.native_expert_layout(t, t, H, I)
    xd = dev(rng.standard_normal((41, H)).astype(np.float32))
    x = xd.cpu().numpy()
    groups, at = [], 0
    for n in sizes:
        groups.append([(at + j) % 41 for j in range(n)])
        at += n
    ids = [i % 2 for i in range(len(groups))]
    out = run_grouped(L, dev(stack_blobs(blobs)), ids, groups, xd, at).cpu().numpy()
    want = {e: O.expert_forward(Lo, blobs[e], x, dtype=np.float64) for e in set(ids)}
    at = 0
    for e, toks in zip(ids, groups):
        assert rel_l2(out[at:at + len(toks)], want[e][toks]) < 4e-4, (e, toks, rel_l2(out[at:at + len(toks)], want[e][toks]))
        at += len(toks)
