"""Decode GEMV with more rows of an expert than one pass over its weights serves (4 or 8 by the rows per expert, 4 in the GGUF
formats): ids that repeat within a token, calls of more than 16 tokens where decode_max_tokens takes them there, and both forms
against one another."""
import numpy as np
import pytest

import oracle
from gfx1151_engine_b200 import synth
from helpers import MAX_ABS_TOL, MEAN_REL_TOL, assert_output_close, bf16_out_to_f32, bf16_tensor, to_bf16_f32
from test_gpu_parity import bits, make_op, run_layer

pytestmark = pytest.mark.gpu


def expert_outputs(spec, layer, x):
    """[experts][T][d]: every expert's output for every token, weight 1."""
    one = synth.LayerSpec(**dict(vars(spec), topk=1, shared=False))
    logits = np.full((spec.experts, len(x), spec.experts), -50.0, np.float32)
    for e in range(spec.experts):
        logits[e, :, e] = 50.0
    return np.stack([oracle.moe_forward(one, layer, x, logits=logits[e])[0] for e in range(spec.experts)])


@pytest.mark.parametrize("T", [1, 2, 5])
@pytest.mark.parametrize("fmt", ["q4cp", "gguf"])
def test_repeated_ids(cuda, fmt, T):
    torch = cuda
    spec = synth.LayerSpec(experts=16, topk=16, d=512, mid=128, fmt=fmt)
    layer = synth.make_layer(spec, seed=96)
    xb = synth.make_x(synth.rng_for(96, 9), T, spec.d)
    y_e = expert_outputs(spec, layer, synth.bf16_bits_to_f32(xb))
    w = synth.rng_for(96, 1).uniform(0.5, 1.5, size=(T, 16)).astype(np.float32)
    w /= w.sum(axis=1, keepdims=True)
    op = make_op(torch, spec, 16, layer=layer)
    for row in ([3] * 16, [3] * 9 + [5] * 5 + [0, 7], [2, 9, 2, 11, 4, 9, 0, 1, 3, 5, 6, 7, 8, 10, 12, 13]):
        ids = np.stack([np.roll(row, t) for t in range(T)]).astype(np.int32)
        out = torch.full((T, spec.d), float("nan"), dtype=torch.bfloat16, device="cuda")
        op.moe_q4w_run(0, bf16_tensor(torch, xb, (T, spec.d)), torch.from_numpy(ids).cuda(), torch.from_numpy(w).cuda(), out)
        op.synchronize()
        want = sum(w[:, s, None] * y_e[ids[:, s], np.arange(T)] for s in range(16))
        assert_output_close(bf16_out_to_f32(torch, out), want, "%s T=%d %r" % (fmt, T, row))
    op.close()


# one launch per GEMM holds 640 passes: (T * 8 + 24 * (rows - 1)) / rows at most
@pytest.mark.parametrize("fmt,T", [("gguf", 40), ("gguf", 311), ("gguf", 330), ("gguf", 700), ("q4cp", 622), ("q4cp", 640), ("q4cp", 1300)])
def test_decode_max_tokens_above_16(cuda, fmt, T):
    torch = cuda
    spec = synth.LayerSpec(experts=24, topk=8, d=256, mid=64, fmt=fmt, shared=fmt == "q4cp")
    layer = synth.make_layer(spec, seed=97)
    xb = synth.make_x(synth.rng_for(97, 9), T, spec.d)
    logits = synth.make_logits(synth.rng_for(97, T), T, spec.experts)
    y_o, ids_o, _ = oracle.moe_forward(spec, layer, synth.bf16_bits_to_f32(xb), logits=logits)
    op = make_op(torch, spec, T, layer=layer, decode_max_tokens=T)
    y = run_layer(torch, op, spec, xb, logits)
    assert np.array_equal(op.get_routing(T)[0][:, :8], ids_o[:, :8])
    assert_output_close(y, y_o, "%s T=%d" % (fmt, T))
    # the fp32 sums of this path, to the bit those of calls of 16
    for t in (0, (T - 16) // 2, T - 16):
        assert np.array_equal(bits(run_layer(torch, op, spec, xb[t:t + 16], logits[t:t + 16])), bits(y[t:t + 16])), t
    op.close()


def test_eight_rows_per_pass_on_few_experts(cuda):
    """Decode calls with many rows per expert make passes of eight rows (q4cp), not of four: 661 of them, two launches per GEMM."""
    torch = cuda
    T, E, k = 640, 24, 8
    spec = synth.LayerSpec(experts=E, topk=k, d=256, mid=64, shared=True)
    op = make_op(torch, spec, T, layer=synth.make_layer(spec, seed=98), decode_max_tokens=T)
    xb, logits = synth.make_x(synth.rng_for(98, 9), T, spec.d), synth.make_logits(synth.rng_for(98, 1), T, E)
    counts = []
    for n in (17, T):
        before = op.launches
        run_layer(torch, op, spec, xb[:n], logits[:n])
        counts.append(op.launches - before)
    op.close()
    passes = (T * k + E * 7) // 8
    assert 640 < passes <= 1280 and counts[1] - counts[0] == 2


# lines between four and eight rows per pass: 5 / 6 tokens (routing inside the GEMV), 22 / 23 (in front of it)
@pytest.mark.parametrize("E,k,d,mid,lengths", [(8, 4, 384, 192, (1, 4, 5, 6, 16)), (8, 4, 2560, 640, (1, 4, 5, 6, 13)),
                                               (32, 4, 1280, 704, (4, 16, 22, 23, 64))])
@pytest.mark.parametrize("shared", [False, True])
def test_four_and_eight_rows_give_the_same_bits(cuda, E, k, d, mid, lengths, shared):
    spec = synth.LayerSpec(experts=E, topk=k, d=d, mid=mid, shared=shared, book="random")
    layer = synth.make_layer(spec, seed=99)
    T = lengths[-1]
    xb = synth.make_x(synth.rng_for(99, 9), T, d)
    logits = synth.make_logits(synth.rng_for(99, 1), T, E)
    logits[:, 3] += 20.0                        # all tokens take this expert
    op = make_op(cuda, spec, T, layer=layer, decode_max_tokens=64)
    y = run_layer(cuda, op, spec, xb, logits)
    y_o, ids_o, _ = oracle.moe_forward(spec, layer, synth.bf16_bits_to_f32(xb), logits=logits)
    assert np.array_equal(op.get_routing(T)[0][:, :k], ids_o[:, :k])
    # the suite's bounds; one bf16 step (2^-7 of the value at most) where outputs are large and an fp16 hidden value crosses a rounding boundary
    ref = to_bf16_f32(y_o)
    diff = np.abs(y - ref)
    assert np.isfinite(y).all() and (diff <= np.maximum(MAX_ABS_TOL, np.abs(ref) * 2.0 ** -7)).all()
    assert diff.mean() <= MEAN_REL_TOL * np.abs(ref).mean()
    for n in lengths[:-1]:
        assert np.array_equal(bits(run_layer(cuda, op, spec, xb[:n], logits[:n])), bits(y[:n])), n
    op.close()
