"""Small kernels inside the one-call step: their blocks are scheduled while the kernel ahead still fills most SMs, and must not pile up on the few
that have room.  What such a kernel takes behind its predecessor, against the same kernel as a plain launch on an empty GPU."""
import re

import pytest
import torch
from torch.profiler import ProfilerActivity, profile

from basalt_b200 import capi, moe

pytestmark = pytest.mark.gpu


def kernels(run, n):
    """(name, start ns, end ns) of every kernel of n runs, by end"""
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as p:
        for _ in range(n):
            run()
        torch.cuda.synchronize()
    ev = [e for e in p.profiler.kineto_results.events() if str(e.device_type()).endswith("CUDA")]
    return sorted(((e.name(), e.start_ns(), e.start_ns() + e.duration_ns()) for e in ev), key=lambda e: e[2])


def median(v):
    return sorted(v)[len(v) // 2]


def behind(make, x, name, before, n=30):
    """from the end of the launch before (a `before`) to the end of kernel `name` in the captured step, and its time as a plain launch, ns"""
    flush = torch.empty(1 << 28, dtype=torch.uint8, device="cuda")        # the weights that such a step streams through L2
    took, layers = {}, []
    for pdl in (True, False):
        layer = make(pdl)
        layer.capture(x)

        def run():
            flush.zero_()
            layer.forward_graphed(x)
        for _ in range(3):
            run()
        torch.cuda.synchronize()
        ev = kernels(run, n)
        at = [i for i, e in enumerate(ev) if re.search(name, e[0])]
        assert len(at) >= n - 1 and all(before in ev[i - 1][0] for i in at)
        took[pdl] = median([ev[i][2] - (ev[i - 1][2] if pdl else ev[i][1]) for i in at])
        layer.check_status()
        layers.append(layer)
    assert torch.equal(layers[0].ids, layers[1].ids) and torch.equal(layers[0].y, layers[1].y)
    return took[True], took[False]


@pytest.mark.parametrize("T", [32, 64])
def test_selection_is_spread(lib, cuda, T):
    """At most 1.4 times (about twice with 36 of 64 tokens on one SM)."""
    H, I, E = 7168, 256, 256
    g = torch.Generator(device="cuda").manual_seed(T)
    gate = torch.randn((E, H), generator=g, device="cuda") * 0.02
    bias = torch.randn(E, generator=g, device="cuda") * 0.01
    x = torch.randn((T, H), generator=g, device="cuda").bfloat16()
    L = moe.native_expert_layout(capi.TYPE_NVFP4, capi.TYPE_NVFP4, H, I)
    blobs = moe.pack_experts(L, torch.zeros((E, L.bytes), dtype=torch.uint8, device="cuda"))
    args = moe.RouterArgs(n_expert=E, n_embd=H, k=8, weight_scale=2.5, gate=capi.GATE_SIGMOID, n_group=8, topk_group=4)
    got, alone = behind(lambda pdl: moe.NativeMoELayer(gate, bias, blobs, L, args, max_tokens=T, packed=True, pdl=pdl), x, "router_select_kernel", "router_logits_kernel")
    assert got < 1.4 * alone, (got, alone)


@pytest.mark.parametrize("t,H,I,k,T", [(capi.TYPE_NVFP4, 7168, 2048, 4, 12), (capi.TYPE_IQ1_M, 7168, 2048, 4, 8)])
def test_swiglu_images_are_spread(lib, cuda, t, H, I, k, T):
    """At most 2.3 times: 3.1 and 2.9 with eight blocks on one SM, 1.7 and 1.8 with four."""
    E = 32
    g = torch.Generator(device="cuda").manual_seed(T)
    gate = torch.randn((E, H), generator=g, device="cuda") * 0.02
    x = torch.randn((T, H), generator=g, device="cuda").bfloat16()
    L = moe.native_expert_layout(t, t, H, I)
    blobs = torch.randint(0, 256, (E + 1, (L.bytes + 15) // 16 * 16), generator=g, device="cuda", dtype=torch.uint8) & 0x37      # small scales, no NaN
    args = moe.RouterArgs(n_expert=E, n_embd=H, k=k, gate=capi.GATE_SOFTMAX)
    got, alone = behind(lambda pdl: moe.NativeMoELayer(gate, None, blobs[:E], L, args, shared_blob=blobs[E], max_tokens=T, pdl=pdl), x, r"(prep|kq)_image_kernel<(0, )?true",
                        "mma_kernel")
    assert got < 2.3 * alone, (got, alone)
