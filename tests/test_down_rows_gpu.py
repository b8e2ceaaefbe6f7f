"""Packed NVFP4 decode where the down product makes its own activation images: n_ff of one and two 256-column chunks, passes of 1 to 8
entries, few passes (one row block a unit) and many (several row blocks a unit, a last unit of fewer).  Each row against the dequantised
expert in 64 bits (bound: the 2e-3 of the packed path), and bit for bit against the same entry in a call of its own."""
import numpy as np
import pytest
import torch

from basalt_b200 import moe
from oracle import oracle as O
from tests.helpers import make_expert_blobs, rel_l2, stack_blobs
from tests.test_packed_gpu import TOL, dev, run_packed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("I", [256, 512])
@pytest.mark.parametrize("H,copies", [(256, 1), (1280, 1), (1280, 50)])
def test_down_rows(lib, cuda, H, I, copies):
    rng = np.random.default_rng(H + I + copies)
    E, T = 5, 24
    Lo, blobs = make_expert_blobs(rng, E, O.T_NVFP4, O.T_NVFP4, H, I)
    L = moe.native_expert_layout(O.T_NVFP4, O.T_NVFP4, H, I)
    packed = moe.pack_experts(L, dev(stack_blobs(blobs)))
    x = rng.standard_normal((T, H)).astype(np.float32)
    x[3] *= 1e-3
    x[5] = 0.0
    xd = dev(x)
    sizes = [1, 8, 9, 0, 17] * copies
    experts = list(range(E)) * copies
    group_tokens = [rng.integers(0, T, s).tolist() for s in sizes]
    out = run_packed(L, packed, experts, group_tokens, xd, n_x_rows=T)
    want = [O.expert_forward(Lo, b, x, dtype=np.float64) for b in blobs]
    at = 0
    for g, (e, toks) in enumerate(zip(experts, group_tokens)):
        for r, t in enumerate(toks):
            row = out[at + r]
            assert not row.any() if not x[t].any() else rel_l2(row, want[e][t]) < TOL, (g, r)
        if toks and g in (0, 1, 4, len(sizes) - 1):
            alone = run_packed(L, packed, [e, e], [toks[-1:], []], xd, n_x_rows=T)
            assert np.array_equal(alone[0].view(np.int32), out[at + len(toks) - 1].view(np.int32)), g
        at += len(toks)
