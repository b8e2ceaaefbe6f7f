"""Q6_K prompt rows where the decoder's copies change: rows of odd and even numbers of 210-byte blocks (every row, or every second block,
starts on 2 bytes), widths that do not fill a tile's 256 weight rows, the last row of a blob (nothing lies behind it), tiles that are not full.
Bound 9e-4: four times the fp16 rounding of weights and SwiGLU rows (2.1e-4 measured)."""
import numpy as np
import pytest
import torch

from basalt_b200 import moe
from oracle import oracle as O
from tests.helpers import make_expert_blobs, rel_l2, stack_blobs
from tests.test_prefill_gpu import run_prefill

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,I,T,E", [(256, 256, 130, 2), (768, 256, 5, 3), (512, 768, 200, 2), (1280, 1280, 70, 2), (256, 2304, 33, 1)])
def test_q6k_prompt_rows(lib, cuda, H, I, T, E):
    rng = np.random.default_rng(H + I)
    Lo, blobs = make_expert_blobs(rng, E, O.T_Q6_K, O.T_Q6_K, H, I)
    L = moe.native_expert_layout(O.T_Q6_K, O.T_Q6_K, H, I)
    ids = rng.integers(0, E, (T, 1)).astype(np.int32)
    xd = torch.from_numpy(rng.standard_normal((T, H)).astype(np.float32)).cuda().bfloat16()
    x = xd.float().cpu().numpy()
    dm, cnt, off, src, _ = run_prefill(L, torch.from_numpy(stack_blobs(blobs)).cuda(), ids, 1, E, xd)
    for e in range(E):
        if cnt[e]:
            want = O.expert_forward(Lo, blobs[e], x[src[off[e]:off[e + 1]]], dtype=np.float64)
            assert rel_l2(dm[off[e]:off[e + 1]], want) < 9e-4, (e, rel_l2(dm[off[e]:off[e + 1]], want))
