"""NVFP4, IQ3_S and (odd numbers of 256-column blocks) IQ1_M experts in place where the streaming kernel's launch shape changes: rows split over four, two or no warps (few, some and
many groups), one block of sixteen warps or two of eight (narrow and wide rows), one codebook copy or sixteen, runs of row blocks that
end inside a pass.  Bound 1e-5, as for the same kernel's other tests: fp16 hi + lo rows (22 bits), fp32 sums over at most 5120 columns.  IQ1_M,
which the fp32 kernels had before: 8e-7, four times the measured 1.9e-7."""
import numpy as np
import pytest

from basalt_b200 import moe
from oracle import oracle as O
from tests.helpers import make_expert_blobs, rel_l2, stack_blobs
from tests.test_experts_gpu import dev, run_grouped

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t,H,I", [(O.T_NVFP4, 2048, 512), (O.T_NVFP4, 4096, 320), (O.T_NVFP4, 512, 3584), (O.T_IQ3_S, 2048, 512), (O.T_IQ3_S, 3072, 512),
                                   (O.T_IQ3_S, 512, 5120), (O.T_IQ1_M, 768, 256), (O.T_IQ1_M, 2560, 1280), (O.T_IQ1_M, 256, 3840), (O.T_IQ1_M, 5120, 768)])
@pytest.mark.parametrize("n_groups", [2, 40, 300])
def test_runs_of_row_blocks(lib, cuda, t, H, I, n_groups):
    rng = np.random.default_rng(H + I + n_groups)
    Lo, blobs = make_expert_blobs(rng, 2, t, t, H, I)
    L = moe.native_expert_layout(t, t, H, I)
    xd = dev(rng.standard_normal((11, H)).astype(np.float32))
    x = xd.cpu().numpy()
    groups = [[(g + j) % 11 for j in range(1 + (g % 7 == 3) * 8)] for g in range(n_groups)]      # one entry, now and then nine
    ids = [g % 2 for g in range(n_groups)]
    out = run_grouped(L, dev(stack_blobs(blobs)), ids, groups, xd, sum(map(len, groups))).cpu().numpy()
    want = [O.expert_forward(Lo, b, x, dtype=np.float64) for b in blobs]
    at = 0
    for e, toks in zip(ids, groups):
        assert rel_l2(out[at:at + len(toks)], want[e][toks]) < (8e-7 if t == O.T_IQ1_M else 1e-5), (e, toks, rel_l2(out[at:at + len(toks)], want[e][toks]))
        at += len(toks)
