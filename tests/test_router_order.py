"""Top-k selection where the order of the logits alone does not give the reference's ids: probabilities that are
denormal or zero floats."""
import numpy as np
import pytest

import gfx1151_engine_b200 as pkg
import oracle
from gfx1151_engine_b200 import synth
from test_gpu_parity import make_op, run_layer

pytestmark = pytest.mark.gpu


def want_ids(logits, k):
    """Largest float probability first, ties to the lowest id."""
    _, w, p = oracle.router_topk(logits, k, want_probs=True)
    return np.argsort(-p, axis=1, kind="stable")[:, :k], w[:, :k]


def check_ids(torch, spec, layer, logits, **kw):
    """ids and weights of a whole call and of router_topk_b."""
    T, k = len(logits), spec.topk
    ids_o, w_o = want_ids(logits, k)
    op = make_op(torch, spec, T, layer=layer, **kw)
    run_layer(torch, op, spec, synth.make_x(synth.rng_for(98, 9), T, spec.d), logits)
    got = [op.get_routing(T)[:2]]
    ids = torch.full((T, 16), -1, dtype=torch.int32, device="cuda")
    w = torch.full((T, 16), -1.0, dtype=torch.float32, device="cuda")
    op.router_topk_b(torch.from_numpy(logits).cuda(), ids, w)
    op.synchronize()
    got.append((ids.cpu().numpy(), w.cpu().numpy()))
    for i, g in got:
        assert np.array_equal(i[:, :k], ids_o)
        assert np.abs(g[:, :k] - w_o).max() <= 1e-6
    op.close()


@pytest.mark.parametrize("decode_impl", [pkg.DECODE_AUTO, pkg.DECODE_FUSED])
@pytest.mark.parametrize("E,k", [(64, 4), (512, 10)])
@pytest.mark.parametrize("T", [1, 5, 13, 77])
def test_widely_spread_logits(cuda, T, E, k, decode_impl):
    """One or some logits far above the others: by 79 to 98 the others' probabilities go from normal through denormal
    floats, beyond 104 they are zero."""
    spec = synth.LayerSpec(experts=E, topk=k, d=128, mid=64)
    layer = synth.make_layer(spec, seed=98)
    for lead in (78.0, 84.0, 92.0, 98.0, 120.0, 200.0):
        logits = synth.make_logits(synth.rng_for(98, T), T, E)
        logits[:, 40] = lead
        if T > 1:
            logits[T // 2, 7:7 + k // 2] = lead - 0.5 - np.arange(k // 2)
        check_ids(cuda, spec, layer, logits, decode_impl=decode_impl)
