"""Calls of more than 16 tokens with few rows per expert on a large layer: experts with as many rows as one pass of the
decode GEMV serves (8, 4 in the GGUF formats) take that, the others the tensor-core kernels beside it -- if the
former are enough: 123 experts of 2560 x 512. Against the oracle on both sides of either line, in every weight format and
through the other entry points, captured in a graph, and what the other tokens of a call may change."""
import numpy as np
import pytest

import gfx1151_engine_b200 as pkg
import oracle
from gfx1151_engine_b200 import synth
from helpers import assert_output_close, bf16_out_to_f32, bf16_tensor
from test_gpu_parity import bits, make_op, run_layer

pytestmark = pytest.mark.gpu
E = 128

# tokens, top-k, rows of the 128 experts
CASES = {
    "some above": (40, 8, [9, 20, 12, 30, 10] + [8] * 15 + [7] + [2] * 5 + [1] * 102),          # 123 of at most 8 rows
    "one expert short": (40, 8, [9] * 6 + [8] * 18 + [2] * 18 + [1] * 86),                    # 122: all on the tensor cores
    "at most 4": (48, 4, [30, 5, 6] + [4] * 5 + [2] * 11 + [1] * 109),                        # 125 of at most 4 rows
    "all": (32, 4, [1] * 128),
    "popular": (200, 4, [200, 200, 150, 65, 17] + [4] * 15 + [1] * 108),                      # wide tiles and narrow ones too
}


def routed_to(T, topk, counts):
    """Logits that give expert e counts[e] rows (sum T * topk, no token twice to one expert), spread over the tokens."""
    left = np.array(counts)
    assert left.sum() == T * topk and left.max() <= T
    lg = np.zeros((T, E), np.float32)
    for t in range(T):
        take = np.argsort(-left, kind="stable")[:topk]
        left[take] -= 1
        lg[t, take] = 8.0 + 0.25 * np.arange(topk)
    assert (left == 0).all()
    return lg


@pytest.fixture(scope="module", params=["q4cp", "gguf"])
def layer(request):
    spec = synth.LayerSpec(experts=E, topk=8, d=2560, mid=512, shared=request.param == "q4cp", fmt=request.param)
    return spec, synth.make_layer(spec, seed=95)


@pytest.mark.parametrize("case", CASES)
def test_against_oracle(cuda, layer, case):
    T, topk, rows = CASES[case]
    spec = synth.LayerSpec(**dict(vars(layer[0]), topk=topk))
    counts = np.array(rows)[np.random.default_rng(T).permutation(E)]
    logits = routed_to(T, topk, counts)
    xb = synth.make_x(synth.rng_for(95, 9), T, spec.d)
    op = make_op(cuda, spec, T, layer=layer[1])
    y = run_layer(cuda, op, spec, xb, logits)
    n = min(T, 48)
    y_o, ids_o, _ = oracle.moe_forward(spec, layer[1], synth.bf16_bits_to_f32(xb[:n]), logits=logits[:n])
    assert np.array_equal(op.get_routing(T)[0][:n, :topk], ids_o[:, :topk])
    assert np.isfinite(y).all()
    assert_output_close(y[:n], y_o, case)
    assert np.array_equal(bits(run_layer(cuda, op, spec, xb, logits)), bits(y))
    op.close()


def test_captured_call_replays_with_new_inputs(cuda, layer):
    torch = cuda
    spec = layer[0]
    T = 40
    op = make_op(torch, spec, T, layer=layer[1])
    xs = [synth.make_x(synth.rng_for(96, i), T, spec.d) for i in range(2)]
    lgs = [routed_to(T, 8, CASES["some above"][2]), synth.make_logits(synth.rng_for(96, 11), T, E)]
    want = [run_layer(torch, op, spec, x, lg) for x, lg in zip(xs, lgs)]
    x, lg = bf16_tensor(torch, xs[0], (T, spec.d)), torch.from_numpy(lgs[0]).cuda()
    out = torch.empty((T, spec.d), dtype=torch.bfloat16, device="cuda")
    st = torch.cuda.Stream()
    st.wait_stream(torch.cuda.current_stream())
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        op.moe_b(0, x, lg, out, stream=st.cuda_stream)
    for i in (1, 0):
        x.copy_(bf16_tensor(torch, xs[i], (T, spec.d)))
        lg.copy_(torch.from_numpy(lgs[i]))
        g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(bits(bf16_out_to_f32(torch, out)), bits(want[i]))
    op.close()


@pytest.mark.parametrize("T,popular,decode_max", [(2560, 0, 0), (2048, 10, 0), (2560, 0, 1300)])
def test_host_call_equals_device_call(cuda, T, popular, decode_max):
    """moe_b_host cuts a call into two ranges, in which every expert has few rows; in the whole call none has, or ten
    have more than one pass of the GEMV serves; or a range is no longer than decode_max_tokens. The bytes are those of one
    call."""
    torch = cuda
    spec = synth.LayerSpec(experts=512, topk=2, d=1024, mid=320)
    op = make_op(torch, spec, T, layer=synth.make_layer(spec, seed=94), decode_max_tokens=decode_max)
    n = T // 2
    left = np.array([6] * popular + [(2 * n - 6 * popular) // (512 - popular)] * (512 - popular))
    left[512 - (2 * n - left.sum()):] += 1
    lg = np.zeros((n, 512), np.float32)
    for t in range(n):
        take = np.argsort(-left, kind="stable")[:2]
        left[take] -= 1
        lg[t, take] = 8.0, 8.5
    assert (left == 0).all()
    x = bf16_tensor(torch, synth.make_x(synth.rng_for(94, 9), T, spec.d), (T, spec.d))
    logits = torch.from_numpy(np.concatenate([lg, lg])).cuda()
    out = torch.empty_like(x)
    op.moe_b(0, x, logits, out)
    op.synchronize()
    host = torch.empty((T, spec.d), dtype=torch.bfloat16).pin_memory()
    op.moe_b_host(0, x.cpu().pin_memory(), logits.cpu().pin_memory(), host, T)
    assert torch.equal(host.view(torch.int16), out.cpu().view(torch.int16))
    op.close()


@pytest.mark.parametrize("gu,dn,d,mid", [(pkg.GGML_Q5_K, pkg.GGML_Q5_1, 2560, 512), (pkg.GGML_IQ4_XS, pkg.GGML_IQ4_XS, 2048, 768),
                                         (pkg.GGML_Q8_0, pkg.GGML_Q8_0, 2048, 640), (pkg.GGML_Q4_K, pkg.GGML_IQ4_NL, 2560, 512)])
def test_weight_formats(cuda, gu, dn, d, mid):
    """125 of 128 experts have at most four rows."""
    T, topk, rows = CASES["at most 4"]
    spec = synth.LayerSpec(experts=E, topk=topk, d=d, mid=mid, fmt="gguf", gg_gu=gu, gg_dn=dn)
    layer = synth.make_layer(spec, seed=97)
    logits = routed_to(T, topk, np.array(rows)[np.random.default_rng(T).permutation(E)])
    xb = synth.make_x(synth.rng_for(97, 9), T, d)
    y_o, _, _ = oracle.moe_forward(spec, layer, synth.bf16_bits_to_f32(xb), logits=logits)
    op = make_op(cuda, spec, T, layer=layer)
    assert_output_close(run_layer(cuda, op, spec, xb, logits), y_o, "%d/%d" % (gu, dn))
    op.close()


def test_other_entry_points(cuda, layer):
    """moe_b_hc adds what moe_b stores; moe_q4w_run with the call's own ids gives its bytes, and with the ids of two tokens out of
    range leaves those tokens zero and the others within the suite's bounds (the experts lose rows)."""
    torch = cuda
    spec = layer[0]
    T, topk, rows = CASES["some above"]
    logits = routed_to(T, topk, rows)
    xb = synth.make_x(synth.rng_for(98, 9), T, spec.d)
    op = make_op(torch, spec, T, layer=layer[1])
    y = run_layer(torch, op, spec, xb, logits)
    ids, w = op.get_routing(T)[:2]
    x, lg = bf16_tensor(torch, xb, (T, spec.d)), torch.from_numpy(logits).cuda()
    state = torch.zeros((T, 4, spec.d), dtype=torch.bfloat16, device="cuda")
    w4 = torch.zeros((T, 4), device="cuda")     # gates of 2 * sigmoid(0) = 1
    op.moe_b_hc(0, x, lg, w4, state)
    op.synchronize()
    assert np.array_equal(bits(bf16_out_to_f32(torch, state)), bits(np.repeat(y[:, None], 4, axis=1)))

    def routed(i):
        out = torch.full((T, spec.d), float("nan"), dtype=torch.bfloat16, device="cuda")
        op.moe_q4w_run(0, x, torch.from_numpy(i).cuda(), torch.from_numpy(w).cuda(), out)
        torch.cuda.synchronize()
        return bf16_out_to_f32(torch, out)
    assert np.array_equal(bits(routed(ids)), bits(y))
    bad = ids.copy()
    bad[[3, 29]] = E + 1
    z = routed(bad)
    with pytest.raises(pkg.B200MoeError):
        op.synchronize()
    keep = np.setdiff1d(np.arange(T), [3, 29])
    assert_output_close(z[keep], y[keep], "others")
    if not spec.shared:
        assert (z[[3, 29]] == 0).all()
    op.close()


def test_neighbours(cuda, layer):
    """Whether an expert's rows take the GEMV depends on the other tokens of the call: a token's output may differ by rounding
    between calls (the suite's bounds), with GEMM_TC it does not."""
    spec = layer[0]
    T = 40
    xb = synth.make_x(synth.rng_for(99, 9), T, spec.d)
    a = routed_to(T, 8, CASES["some above"][2])
    b = a.copy()
    b[20:] = 0.0
    b[20:, :8] = 8.0 + 0.25 * np.arange(8)    # popular experts: fewer than 123 are left for the GEMV
    for impl in (pkg.GEMM_AUTO, pkg.GEMM_TC):
        op = make_op(cuda, spec, T, layer=layer[1], impl=impl)
        ya, yb = run_layer(cuda, op, spec, xb, a)[:20], run_layer(cuda, op, spec, xb, b)[:20]
        assert_output_close(ya, yb, "impl %d" % impl)
        if impl == pkg.GEMM_TC:
            assert np.array_equal(bits(ya), bits(yb))
            assert np.array_equal(bits(run_layer(cuda, op, spec, xb[:7], a[:7])), bits(ya[:7]))
        op.close()
