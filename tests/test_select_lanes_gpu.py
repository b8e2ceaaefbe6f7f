"""Selection by one warp.  Softmax where the winners crowd: all values of one lane (experts e, e + 32, ...) first, more winners than a lane holds, equal
values, experts of probability zero, for each number of values a lane has.  Ids against the rank rule (value descending, index ascending) on
logits whose order no rounding can change; weights against 64 bits (bound 1e-5: an expf and a division of 32 bits each)."""
import numpy as np
import pytest
import torch

from basalt_b200 import capi, moe

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E", [64, 128, 256, 384, 512, 640, 1024])
def test_crowded_lanes(lib, cuda, E):
    rng = np.random.default_rng(E)
    k = 32
    lg = np.full((4, E), -60.0, np.float32)
    lane5 = np.arange(5, E, 32)
    for t, lead in enumerate((lane5, lane5[::-1], np.concatenate([lane5, np.arange(0, E, 32)]), rng.permutation(E))):
        lead = lead[:40]
        lg[t, lead] = 4.0 - 0.25 * np.arange(len(lead))
    lg[2, lane5[:2]] = 4.5                       # equal values of one lane
    lg[0, 6] = -np.inf
    p = np.exp(lg.astype(np.float64) - lg.max(1, keepdims=True))
    want = np.argsort(-p, axis=1, kind="stable")[:, :k]
    for kind in (capi.GATE_SOFTMAX, capi.GATE_SOFTMAX_FAST):
        ids, w = moe.router_select(torch.from_numpy(lg).cuda(), None, moe.RouterArgs(n_expert=E, k=k, gate=kind))
        assert np.array_equal(ids.cpu().numpy(), want), kind
        top = np.take_along_axis(p, want, 1)
        assert np.abs(w.cpu().numpy() - top / top.sum(1, keepdims=True)).max() < (1e-5 if kind == capi.GATE_SOFTMAX else 1e-3)


@pytest.mark.parametrize("E", [64, 256, 512])
@pytest.mark.parametrize("kind", [capi.GATE_SIGMOID, capi.GATE_SQRT_SOFTPLUS])
def test_a_token_of_nan_logits(lib, cuda, E, kind):
    """No score compares, so the ids are the ones that lane 0 offers, its own experts (0, 32, ...) and then none; in both selection kernels.  The
    other tokens keep theirs."""
    rng = np.random.default_rng(E)
    lg = rng.standard_normal((12, E)).astype(np.float32)
    a = moe.RouterArgs(n_expert=E, k=6, gate=kind)
    sound, _ = moe.router_select(torch.from_numpy(lg).cuda(), None, a)
    want = sound.cpu().numpy()
    lg[5] = np.nan
    want[5] = [32 * r if 32 * r < E else -1 for r in range(6)]
    l = torch.from_numpy(lg).cuda()
    table = torch.arange(1, E + 1, dtype=torch.int64, device="cuda") * 256       # addresses that the plan only copies
    for ids, w in (moe.router_select(l, None, a), moe.route_plan(l, None, a, table)[:2]):
        assert np.array_equal(ids.cpu().numpy(), want)
        w = w.cpu().numpy()
        assert np.isnan(w[5]).all() and np.isfinite(np.delete(w, 5, 0)).all()
