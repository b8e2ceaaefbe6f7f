"""A window's selection inside the one-call step: its blocks are scheduled while the logits kernel still runs, and must not pile up on the few
SMs that have room then.  From the last logit to the selection's end may take at most 1.4 times what the selection takes as a plain launch on
an empty GPU (about twice as much with 36 of 64 tokens on one SM)."""
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


@pytest.mark.parametrize("T", [32, 64])
def test_selection_is_spread(lib, cuda, T):
    H, I, E, n = 7168, 256, 256, 30
    g = torch.Generator(device="cuda").manual_seed(T)
    gate = torch.randn((E, H), generator=g, device="cuda") * 0.02
    bias = torch.randn(E, generator=g, device="cuda") * 0.01
    x = torch.randn((T, H), generator=g, device="cuda").bfloat16()
    L = moe.native_expert_layout(capi.TYPE_NVFP4, capi.TYPE_NVFP4, H, I)
    blobs = moe.pack_experts(L, torch.zeros((E, L.bytes), dtype=torch.uint8, device="cuda"))
    args = moe.RouterArgs(n_expert=E, n_embd=H, k=8, weight_scale=2.5, gate=capi.GATE_SIGMOID, n_group=8, topk_group=4)
    flush = torch.empty(1 << 28, dtype=torch.uint8, device="cuda")        # the weights that such a step streams through L2
    ids, took = [], {}
    for pdl in (True, False):
        layer = moe.NativeMoELayer(gate, bias, blobs, L, args, max_tokens=T, packed=True, pdl=pdl)
        layer.capture(x)

        def run():
            flush.zero_()
            layer.forward_graphed(x)
        for _ in range(3):
            run()
        torch.cuda.synchronize()
        ev = kernels(run, n)
        at = [i for i, e in enumerate(ev) if "router_select_kernel" in e[0]]
        assert len(at) >= n - 1 and all("router_logits_kernel" in ev[i - 1][0] for i in at)
        took[pdl] = median([ev[i][2] - (ev[i - 1][2] if pdl else ev[i][1]) for i in at])
        layer.check_status()
        ids.append(layer.ids.clone())
    assert torch.equal(*ids)
    assert took[True] < 1.4 * took[False], took
