"""The streaming tensor-core kernel's formats and widths under every row kind, output type and SwiGLU form, against the warp-per-row fp32
kernel over the same rows.  Bound 1e-5 (two fp16 terms a row; fp32 sums of at most 640 products); bf16 outputs are two roundings of
nearly the same number: 2^-8 / sqrt(3) where they fall apart, which fewer than one in a hundred does."""
import numpy as np
import pytest
import torch

from basalt_b200 import moe
from oracle import oracle as O
from tests.helpers import make_expert_blobs, rel_l2, stack_blobs
from tests.test_experts_gpu import dev, run_grouped

pytestmark = pytest.mark.gpu
PLAIN = 4


@pytest.mark.parametrize("t,H,I", [(O.T_IQ3_S, 512, 512), (O.T_NVFP4, 512, 640), (O.T_NVFP4, 256, 192), (O.T_NVFP4, 256, 512)])
@pytest.mark.parametrize("act", ["f32", "bf16", "q8_1"])
@pytest.mark.parametrize("form", ["silu", "limit", "softcap"])
@pytest.mark.parametrize("out", [torch.float32, torch.bfloat16])
def test_options(lib, cuda, t, H, I, act, form, out):
    rng = np.random.default_rng(H + I)
    _, blobs = make_expert_blobs(rng, 2, t, t, H, I)
    plain = moe.native_expert_layout(t, t, H, I)
    L = moe.native_expert_layout(t, t, H, I, **{"silu": {}, "limit": {"swiglu_limit": 0.2}, "softcap": {"gate_softcap": 0.5, "up_softcap": 0.4}}[form])
    xd = dev(rng.standard_normal((9, H)).astype(np.float32))
    if act != "f32":
        xd = xd.bfloat16() if act == "bf16" else moe.quantize_q8_1_rows(xd)
    bd, groups = dev(stack_blobs(blobs)), [[8], list(range(9))]
    got = run_grouped(L, bd, [1, 0], groups, xd, 10, out).float().cpu().numpy()
    L.options = PLAIN
    want = run_grouped(L, bd, [1, 0], groups, xd, 10, out).float().cpu().numpy()
    assert rel_l2(got, want) < (1e-5 if out == torch.float32 else 2 ** -8 / 3 ** 0.5 / 10)
    if form != "silu":
        assert rel_l2(want, run_grouped(plain, bd, [1, 0], groups, xd, 10, out).float().cpu().numpy()) > 1e-2      # the form bites
