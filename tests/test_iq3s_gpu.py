"""IQ3_S experts on the streaming tensor-core kernel at the sizes where its row tiles, its 512-column chunks and its passes begin
and end, against the warp-per-row kernel's own oracle.  Bound 1e-5: weights are exact integers times the block's fp16 scale, rows
enter as fp16 hi + lo terms (22 bits) and every product is summed in fp32 over at most 2048 columns."""
import numpy as np
import pytest

from basalt_b200 import moe
from oracle import oracle as O
from tests.helpers import make_expert_blobs, rel_l2, stack_blobs
from tests.test_experts_gpu import dev, run_grouped

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,I", [(512, 512), (2048, 512), (512, 1536), (1536, 1024)])
@pytest.mark.parametrize("act", ["f32", "bf16"])
def test_iq3s_rows(lib, cuda, H, I, act):
    rng = np.random.default_rng(H + I)
    Lo, blobs = make_expert_blobs(rng, 3, O.T_IQ3_S, O.T_IQ3_S, H, I)
    L = moe.native_expert_layout(O.T_IQ3_S, O.T_IQ3_S, H, I)
    xd = dev(rng.standard_normal((13, H)).astype(np.float32))
    if act == "bf16":
        xd = xd.bfloat16()
    x = xd.float().cpu().numpy()
    groups = [[4], list(range(13)), [0, 7]]          # one entry, more than one pass, fewer than a pass
    out = run_grouped(L, dev(stack_blobs(blobs)), [2, 0, 1], groups, xd, 16).cpu().numpy()
    at = 0
    for e, toks in zip([2, 0, 1], groups):
        want = O.expert_forward(Lo, blobs[e], x[toks], dtype=np.float64)
        assert rel_l2(out[at:at + len(toks)], want) < 1e-5, (e, rel_l2(out[at:at + len(toks)], want))
        at += len(toks)
