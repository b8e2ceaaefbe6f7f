"""NVFP4 experts whose down rows are not whole 256-column chunks: the streaming tensor-core kernel at the widths where its last
chunk, its copies' width (16, 8 or 4 bytes) or its row tiles change.  Bound 1e-5: rows enter as fp16 hi + lo terms (22 bits) and
every product is summed in fp32 over at most 2048 columns."""
import numpy as np
import pytest

from basalt_b200 import moe
from oracle import oracle as O
from tests.helpers import make_expert_blobs, rel_l2, stack_blobs
from tests.test_experts_gpu import dev, run_grouped

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,I", [(256, 64), (512, 128), (256, 192), (512, 320), (2048, 448), (2560, 640), (256, 960), (512, 512)])
@pytest.mark.parametrize("act", ["f32", "bf16"])
def test_down_rows_of_any_block_count(lib, cuda, H, I, act):
    rng = np.random.default_rng(H + I)
    Lo, blobs = make_expert_blobs(rng, 3, O.T_NVFP4, O.T_NVFP4, H, I)
    L = moe.native_expert_layout(O.T_NVFP4, O.T_NVFP4, H, I)
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
