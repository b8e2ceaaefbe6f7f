"""Decode experts in place over rows whose values reach the ends of fp32: the streaming tensor-core kernel, which takes a row as fp16
terms under a power of two, against the warp-per-row fp32 kernel, each product by itself.  The same results are infinite and NaN;
finite ones agree to 1e-5 (two terms hold 22 bits of a row, the fp32 kernel sums at most 1280 products)."""
import numpy as np
import pytest
import torch

from basalt_b200 import moe
from oracle import oracle as O
from tests.helpers import make_expert_blobs, rel_l2, stack_blobs
from tests.test_experts_gpu import dev

pytestmark = pytest.mark.gpu
STAGE_GU, STAGE_DOWN, PLAIN = 1, 2, 4
SHAPES = [(O.T_IQ3_S, 512, 512), (O.T_IQ3_S, 512, 1024), (O.T_NVFP4, 512, 320), (O.T_NVFP4, 1280, 192), (O.T_NVFP4, 512, 512),
          (O.T_IQ1_M, 1280, 1280), (O.T_IQ1_M, 2048, 768)]


def rows(rng, K, names):
    x = rng.standard_normal((len(names), K)).astype(np.float32)
    for i, name in enumerate(names):
        if "inf" in name:
            x[i, 7] = -np.inf if name == "minus inf" else np.inf
        if name == "inf and large":
            x[i, 3], x[i, 100] = -1e30, 2.5e30
        if name == "two infs":
            x[i, K - 1] = np.inf
        if name == "nan":
            x[i, 64] = np.nan
        if name.startswith("2^"):
            x[i] = np.ldexp(x[i], int(name[2:]))
        if name in ("largest", "zero"):
            x[i] = 0
        if name == "largest":
            x[i, 5], x[i, 90] = 3.3e38, 1e35        # (a value below 2^-38 of its row's largest would lie under both terms' last bit)
    return x


def run(L, bd, n, x, h, stage):
    """one expert over n rows: the h a gate/up call leaves, or the output of a down call over the given h"""
    dv = dict(device="cuda")
    L.options = stage
    scratch = torch.zeros(moe.native_expert_scratch_bytes(L, n), dtype=torch.uint8, **dv)
    hv = scratch[:n * L.n_ff * 4].view(torch.float32).view(n, L.n_ff)
    if h is not None:
        hv.copy_(h)
    out = torch.zeros((n, L.n_embd), **dv)
    i32 = dict(dtype=torch.int32, **dv)
    ent = torch.arange(n, **i32)
    moe.native_expert_grouped(L, torch.tensor([bd.data_ptr(), 0], dtype=torch.int64, **dv), torch.tensor([0, n, n], **i32), torch.ones(1, **i32), ent, ent, 1, n, x,
                              scratch, out)
    torch.cuda.synchronize()
    return (hv if stage & STAGE_GU else out).cpu().numpy().copy()


def same(names, got, want):
    for i, name in enumerate(names):
        g, w = got[i], want[i]
        assert np.array_equal(np.isnan(g), np.isnan(w)) and np.array_equal(np.isinf(g), np.isinf(w)), name
        assert np.array_equal(np.sign(g[np.isinf(g)]), np.sign(w[np.isinf(w)])), name
        f = np.isfinite(w)
        assert not f.any() or rel_l2(g[f], w[f]) < 1e-5, (name, rel_l2(g[f], w[f]))


@pytest.mark.parametrize("t,H,I", SHAPES)
@pytest.mark.parametrize("act", ["f32", "bf16"])
def test_gate_up(lib, cuda, t, H, I, act):
    rng = np.random.default_rng(H + I)
    _, blobs = make_expert_blobs(rng, 1, t, t, H, I)
    L = moe.native_expert_layout(t, t, H, I)
    names = ("plain", "inf", "inf and large", "minus inf", "two infs", "nan", "2^-30", "2^-55", "zero")
    xd = dev(rows(rng, H, names))
    if act == "bf16":
        xd = xd.bfloat16()
    bd = dev(stack_blobs(blobs))
    want = run(L, bd, len(names), xd, None, STAGE_GU | PLAIN)
    assert np.isinf(want[1]).any() and np.isfinite(want[7]).all() and np.abs(want[7]).max() > 0
    same(names, run(L, bd, len(names), xd, None, STAGE_GU), want)


@pytest.mark.parametrize("t,H,I", SHAPES)
def test_down(lib, cuda, t, H, I):
    rng = np.random.default_rng(H + 3 * I)
    _, blobs = make_expert_blobs(rng, 1, t, t, H, I)
    L = moe.native_expert_layout(t, t, H, I)
    names = ("plain", "inf", "inf and large", "minus inf", "two infs", "nan", "2^-86", "2^-100", "2^-110", "2^-122", "largest", "zero")
    h, bd = dev(rows(rng, I, names)), dev(stack_blobs(blobs))
    xd = torch.zeros((len(names), H), device="cuda")
    want = run(L, bd, len(names), xd, h, STAGE_DOWN | PLAIN)
    assert np.isinf(want[1]).any() and np.isfinite(want[9]).all() and np.abs(want[9]).max() > 0
    same(names, run(L, bd, len(names), xd, h, STAGE_DOWN), want)
