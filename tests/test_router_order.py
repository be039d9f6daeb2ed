"""Top-k selection where the order of the logits alone does not give the reference's ids: probabilities that are
denormal or zero floats, many leaders in few residues mod 32, equal and masked (-inf) logits."""
import numpy as np
import pytest

import gfx1151_engine_b200 as pkg
import oracle
from gfx1151_engine_b200 import synth
from helpers import assert_output_close, bf16_out_to_f32, bf16_tensor, dev_bytes
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


@pytest.mark.parametrize("T", [1, 5, 16])
def test_near_tie_among_many_leaders(cuda, T):
    """Hidden states, T <= 16: 48 leaders in three residues mod 32. Expert 40's logit stands on a rounding boundary: added
    in index order it is 1, as expert 8's, which then goes first; added as a tree it is the next larger float."""
    torch = cuda
    spec = synth.LayerSpec(experts=512, topk=3, d=128, mid=64, router=True)
    layer = synth.make_layer(spec, seed=99)
    w = np.zeros((512, 128), np.float32)
    w[:, 0] = -(1.0 + np.arange(512)) / 512
    lead = [e for e in range(512) if e % 32 in (8, 9, 10)]
    w[lead, 0] = (128.0 + np.arange(len(lead))) / 256
    w[10, 0], w[9, 0], w[8, 0] = 1.5, 1.25, 1.0
    w[40] = 2.0 ** -54
    w[40, :2] = 1.0, 2.0 ** -24
    layer["router_w"] = synth.f32_to_bf16_bits(w)
    assert np.array_equal(synth.bf16_bits_to_f32(layer["router_w"])[lead], w[lead])
    x = np.ones((T, 128), np.float32) * (2.0 ** (np.arange(T) % 3)).astype(np.float32)[:, None]
    x[T // 2, 127] = 1.5
    xb = synth.f32_to_bf16_bits(x)
    y_o, ids_o, _ = oracle.moe_forward(spec, layer, x)
    assert ids_o[0, :3].tolist() == [10, 9, 8]
    op = make_op(torch, spec, T, layer=layer)
    op.load_router(0, dev_bytes(torch, layer["router_w"]))
    out = torch.full((T, spec.d), float("nan"), dtype=torch.bfloat16, device="cuda")
    op.moe_hidden(0, bf16_tensor(torch, xb, (T, spec.d)), out)
    op.synchronize()
    assert np.array_equal(op.get_routing(T)[0][:, :3], ids_o[:, :3])
    assert_output_close(bf16_out_to_f32(torch, out), y_o, "T=%d" % T)
    op.close()


def tied(kind, T, E):
    lg = synth.make_logits(synth.rng_for(97, T), T, E)
    if kind == "bf16":
        return synth.bf16_bits_to_f32(synth.f32_to_bf16_bits(lg))
    if kind == "eighths":
        return np.round(lg * 8).astype(np.float32) / 8
    if kind == "masked":      # half of the experts
        return np.where(np.arange(E) % 2 == np.arange(T)[:, None] % 2, lg, -np.inf).astype(np.float32)
    if kind == "few left":    # as many as are selected, one more, one less
        left = 8 + np.arange(T)[:, None] % 3 - 1
        return np.where(np.arange(E) * 5 % E < left, lg, -np.inf).astype(np.float32)
    if kind == "adjacent":    # a few floats apart: their probabilities share one
        return (np.float32(0.44) + np.float32(2.0) ** -25 * (np.arange(E) * 7 % 11 + np.arange(T)[:, None] % 5)).astype(np.float32)
    return np.full((T, E), 0.25, np.float32)


@pytest.mark.parametrize("kind", ["bf16", "eighths", "masked", "few left", "adjacent", "equal"])
@pytest.mark.parametrize("T,E,k", [(1, 64, 8), (16, 64, 8), (16, 512, 16), (7, 12, 8), (77, 512, 8)])
def test_equal_and_masked_logits(cuda, T, E, k, kind):
    spec = synth.LayerSpec(experts=E, topk=k, d=128, mid=64)
    check_ids(cuda, spec, synth.make_layer(spec, seed=98), tied(kind, T, E))


@pytest.mark.parametrize("kind", ["zero rows", "zero router", "pairs", "all equal", "near"])
@pytest.mark.parametrize("T,E,k", [(1, 64, 8), (5, 64, 8), (16, 64, 8), (16, 512, 16), (3, 20, 16)])
def test_equal_logits_from_hidden_states(cuda, T, E, k, kind):
    """Rows of zeros (padding), equal rows of the router, and rows that differ in one small element: logits a few floats apart."""
    torch = cuda
    spec = synth.LayerSpec(experts=E, topk=k, d=256, mid=64, router=True)
    layer = synth.make_layer(spec, seed=100)
    x = synth.bf16_bits_to_f32(synth.make_x(synth.rng_for(100, T), T, spec.d)).copy()
    w = synth.bf16_bits_to_f32(layer["router_w"]).copy()
    if kind == "zero rows":
        x[::2] = 0
    if kind == "zero router":
        w[:] = 0
    if kind == "pairs":
        w[1::2] = w[::2]
    if kind in ("all equal", "near"):
        w[:] = w[3]
    if kind == "near":
        x[:, 17] = 1.0
        w[:, 17] = np.float32(2.0) ** -26 * (np.arange(E) * 7 % 11)
    layer["router_w"] = synth.f32_to_bf16_bits(w)
    xb = synth.f32_to_bf16_bits(x)
    ids_o, _ = want_ids(oracle.router_logits(layer["router_w"], x), k)
    op = make_op(torch, spec, T, layer=layer)
    op.load_router(0, dev_bytes(torch, layer["router_w"]))
    out = torch.full((T, spec.d), float("nan"), dtype=torch.bfloat16, device="cuda")
    op.moe_hidden(0, bf16_tensor(torch, xb, (T, spec.d)), out)
    op.synchronize()
    assert np.array_equal(op.get_routing(T)[0][:, :k], ids_o)
    assert torch.isfinite(out).all()
    op.close()
