"""Calls of the grouped GEMMs run tiles of at most 64 rows in the form for few rows (weights through a ring of bulk
copies) and larger ones in the wide form, on two lists side by side or on one, by the call's sizes and the rows of all experts; popular
experts' down GEMM runs on expanded weights. Against the oracle where those forms can go wrong -- K block counts that are odd, one, or
fewer than the ring's stages, experts whose rows end just behind a tile, every weight format -- and bit for bit
against one another on both sides of the rules: a row's sums do not depend on the tile it is in. The rules' lines are read from the
sources, and each call is checked to lie on the side that it stands for."""
import os
import re

import numpy as np
import pytest

import gfx1151_engine_b200 as pkg
import oracle
from gfx1151_engine_b200 import synth
from helpers import assert_output_close, bf16_out_to_f32, bf16_tensor
from oracle import i4r
from test_gpu_parity import bits, make_op, run_layer
from test_i4r_gpu import make_i4r_op, run as run_i4r

pytestmark = pytest.mark.gpu

CSRC = os.path.join(os.path.dirname(pkg.__file__), "csrc")
SOURCES = "".join(open(os.path.join(CSRC, f)).read() for f in ("api.cu", "kernels.h", "tc.h", "common.cuh"))


def line(name):
    """The value of a constant of the rules."""
    return int(re.search(r"\b%s = (\d+)" % name, SOURCES).group(1))


WIDE_ROWS, FEW_ROWS = line("kTcTileN"), line("kTcNarrowN")


def form(E, k, d, mid, T):
    """What a tensor-core call of T > 16 tokens runs: "few" (one list of tiles of 64 rows), "wide" (one of 192), or "both" (the
    device chooses: two launches more)."""
    few, second = T * k <= line("kFewRows") * E, line("kSecondListCycles") * 148 * 8192 // (3 * d * mid)
    if (line("kTileCostFew") * 2 * T * k > (2 * FEW_ROWS + 1) * second) if few else E * d * mid >= line("kBothLists"):
        return "both"
    return "few" if few or (T <= line("kOneListTokens") and T * k <= line("kOneListRows") * E) else "wide"


def device_choice(counts, d, mid):
    """Where the device chooses: the form that it takes for these experts' rows."""
    wide_cost, few_cost = line("kTileCostWide"), line("kTileCostFew")
    wide, few = sum(-(-c // WIDE_ROWS) for c in counts), sum(-(-c // FEW_ROWS) for c in counts)
    ragged = sum(0 < c % WIDE_ROWS <= FEW_ROWS for c in counts)
    both = wide_cost * (wide - ragged) + few_cost * ragged + line("kSecondListCycles") * 148 * 8192 // (3 * d * mid)
    if few_cost * few <= min(wide_cost * wide, both):
        return "few"
    return "wide" if wide_cost * wide <= both else "both"


def popular(logits, experts):
    """All tokens take these experts (in addition to others): as many rows as the call has tokens."""
    logits[:, list(experts)] += 20.0
    return logits


@pytest.mark.parametrize("T", [17, 64, 65, 129])
@pytest.mark.parametrize("shape", [dict(experts=64, topk=2, d=128, mid=64, shared=True, book="random"),
                                   dict(experts=64, topk=4, d=384, mid=192, shared=True),
                                   dict(experts=48, topk=4, d=2560, mid=640, shared=False, book="random")])
def test_narrow_tiles_against_oracle(cuda, shape, T):
    spec = synth.LayerSpec(**shape)
    assert T * spec.topk <= 12 * spec.experts
    layer = synth.make_layer(spec, seed=81)
    logits = popular(synth.make_logits(synth.rng_for(81, T), T, spec.experts), [3])
    xb = synth.make_x(synth.rng_for(81, 9), T, spec.d)
    op = make_op(cuda, spec, T, layer=layer)
    y = run_layer(cuda, op, spec, xb, logits)
    y_o, ids_o, _ = oracle.moe_forward(spec, layer, synth.bf16_bits_to_f32(xb), logits=logits)
    assert np.array_equal(op.get_routing(T)[0][:, :spec.topk], ids_o[:, :spec.topk])
    assert_output_close(y, y_o, "narrow %r T=%d" % (shape, T))
    op.close()


# the last calls of tiles of 64 rows alone, by the rows per expert and by the tokens; one token more runs the wide form alone
@pytest.mark.parametrize("E,T", [(32, 384), (64, 512)])
def test_both_sides_of_the_rule_agree(cuda, E, T):
    spec = synth.LayerSpec(experts=E, topk=4, d=512, mid=256, shared=True)
    assert [form(E, 4, 512, 256, n) for n in (T, T + 1)] == ["few", "wide"]
    layer = synth.make_layer(spec, seed=82)
    logits = popular(synth.make_logits(synth.rng_for(82, 1), T + 1, spec.experts, zipf=True), [5, 17])
    xb = synth.make_x(synth.rng_for(82, 9), T + 1, spec.d)
    op = make_op(cuda, spec, T + 1, layer=layer)
    wide = run_layer(cuda, op, spec, xb, logits)
    narrow = run_layer(cuda, op, spec, xb[:T], logits[:T])
    assert np.array_equal(bits(narrow), bits(wide[:T]))
    op.close()


@pytest.mark.parametrize("types", [(pkg.GGML_Q4_K, pkg.GGML_Q5_1), (pkg.GGML_Q5_K, pkg.GGML_Q5_1), (pkg.GGML_Q8_0, pkg.GGML_Q8_0),
                                   (pkg.GGML_IQ4_XS, pkg.GGML_IQ4_XS)])
def test_narrow_gguf_equals_wide(cuda, types):
    """The GGUF images (more metadata per tile, two planes for Q8_0): the same rows in a call of the few-row and in one of the wide form."""
    torch = cuda
    E, k, d, mid = 16, 2, 512, 256
    gen = np.random.default_rng(83)
    size = {pkg.GGML_Q4_K: (256, 144), pkg.GGML_Q5_K: (256, 176), pkg.GGML_Q5_1: (32, 24), pkg.GGML_Q8_0: (32, 34), pkg.GGML_IQ4_XS: (256, 136)}

    def blocks(rows, cols, t):
        per, n = size[t]
        b = gen.integers(0, 256, size=(rows * cols // per, n), dtype=np.uint8)
        scale = 2e-5 if t == pkg.GGML_IQ4_XS else 1e-3 if per == 256 else 1e-2
        b[:, 0:2] = np.full(len(b), scale, "<f2").view(np.uint8).reshape(-1, 2)
        if t not in (pkg.GGML_Q8_0, pkg.GGML_IQ4_XS):
            b[:, 2:4] = np.full(len(b), 5e-4 if per == 256 else -1e-1, "<f2").view(np.uint8).reshape(-1, 2)
        return torch.from_numpy(b.reshape(-1)).cuda()

    T = 600
    assert form(E, k, d, mid, T) == "wide" and form(E, k, d, mid, 90) == "few"
    op = pkg.MoeOperator(E, k, d, mid, T)
    op.load_gguf(0, blocks(E * mid, d, types[0]), blocks(E * mid, d, types[0]), blocks(E * d, mid, types[1]),
                 type_gu=types[0], type_dn=types[1])
    x = torch.randn(T, d, device="cuda").bfloat16()
    logits = torch.randn(T, E, device="cuda")
    out = torch.full((T, d), float("nan"), dtype=torch.bfloat16, device="cuda")
    op.moe_b(0, x, logits, out)
    few = torch.full((90, d), float("nan"), dtype=torch.bfloat16, device="cuda")
    op.moe_b(0, x[:90].contiguous(), logits[:90].contiguous(), few)
    op.synchronize()
    assert torch.isfinite(out.float()).all() and torch.equal(few, out[:90])
    op.close()


@pytest.mark.parametrize("T", [40, 200])
def test_captured_call_replays(cuda, T):
    """The chain's overlapping launches (and the shared expert's launch beside the routed one) in a CUDA
    graph: replays with new inputs in the same buffers give what plain calls give."""
    torch = cuda
    spec = synth.LayerSpec(experts=16, topk=4, d=512, mid=256, shared=True)
    layer = synth.make_layer(spec, seed=84)
    op = make_op(torch, spec, T, layer=layer)
    x = torch.randn(T, spec.d, device="cuda").bfloat16()
    logits = torch.randn(T, spec.experts, device="cuda")
    out = torch.empty(T, spec.d, dtype=torch.bfloat16, device="cuda")
    op.moe_b(0, x, logits, out)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        op.moe_b(0, x, logits, out, stream=torch.cuda.current_stream().cuda_stream)
    for _ in range(3):
        x.copy_(torch.randn(T, spec.d, device="cuda"))
        logits.copy_(torch.randn(T, spec.experts, device="cuda"))
        out.fill_(float("nan"))
        graph.replay()
        replayed = out.clone()
        op.moe_b(0, x, logits, out)
        op.synchronize()
        assert torch.equal(replayed, out)
    del graph
    op.close()


def ids_of_counts(E, k, T, counts):
    """[T][16] distinct ids: expert e < len(counts) gets counts[e] tokens, the others share what is left."""
    left, ids, rest = list(counts), np.zeros((T, 16), np.int32), len(counts)
    for t in range(T):
        # experts that need every token still to come first, then the fullest
        pick = sorted((e for e in range(len(left)) if left[e] > 0), key=lambda e: -left[e])[:k]
        for e in pick:
            left[e] -= 1
        while len(pick) < k:
            pick.append(rest)
            rest = len(counts) + (rest + 1 - len(counts)) % (E - len(counts))
        ids[t, :k] = pick
    assert not any(left)
    return ids


# Calls of T = 12*E/k tokens on a layer of 4096 x 1024, where the device chooses: no expert over a small tile (64 rows) or four just over one
# (tiles of 64 rows alone), 16 just over one or a few of all tokens (two lists), and a few of all tokens with hardly any others (wide
# tiles alone), with rows on both sides of a small tile and of a full one (192)
@pytest.mark.parametrize("fmt", ["q4cp", "i4r"])
def test_both_forms_in_one_call(cuda, fmt):
    """Tiles of more than 64 rows run in the wide form, the others of the same call in the few-row one, or all in either: bit for
    bit the rows of a longer call, which runs the wide form alone."""
    torch = cuda
    E, k, d, mid = 96, 4, 4096, 1024
    T = 12 * E // k
    whole = line("kOneListTokens") + 1
    assert form(E, k, d, mid, T) == "both" and form(E, k, d, mid, whole) == "wide"
    if fmt == "i4r":
        L = synth.make_i4r_layer(E, d, mid, seed=87)
        op = make_i4r_op(torch, E, k, d, mid, whole, L)
    else:
        spec = synth.LayerSpec(experts=E, topk=k, d=d, mid=mid, shared=True)
        op = make_op(torch, spec, whole, layer=synth.make_layer(spec, seed=87))
    w = synth.rng_for(87, 1).uniform(0.2, 1.0, size=(whole, 16)).astype(np.float32) / k
    xb = synth.make_x(synth.rng_for(87, 9), whole, d)
    for counts, choice in (([64, 64], "few"), ([65] * 4, "few"), ([65] * 16, "both"), ([288] * 3, "both"),
                           ([288, 257, 257, 257], "both"), ([288] * 4, "wide"), ([288, 288, 193, 193, 65, 64, 49, 12], "wide")):
        ids = ids_of_counts(E, k, T, counts)
        assert device_choice(np.bincount(ids[:, :k].reshape(-1), minlength=E), d, mid) == choice, counts
        ids = np.concatenate([ids, np.repeat(ids[-1:], whole - T, axis=0)])
        outs = []
        for n in (T, whole):
            before = op.launches
            out = torch.full((n, d), float("nan"), dtype=torch.bfloat16, device="cuda")
            op.moe_q4w_run(0, bf16_tensor(torch, xb[:n], (n, d)), torch.from_numpy(ids[:n]).cuda(), torch.from_numpy(w[:n]).cuda(), out)
            op.synchronize()
            outs.append((bf16_out_to_f32(torch, out), op.launches - before))
        assert np.isfinite(outs[0][0]).all() and np.array_equal(bits(outs[0][0]), bits(outs[1][0][:T])), counts
        assert outs[0][1] == outs[1][1] + 2    # the second list's launch in both GEMM stages
    # captured: the launches beside each other, replayed with the last ids
    x, i_dev, w_dev = bf16_tensor(torch, xb[:T], (T, d)), torch.zeros(T, 16, dtype=torch.int32, device="cuda"), torch.from_numpy(w[:T]).cuda()
    out = torch.full((T, d), float("nan"), dtype=torch.bfloat16, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        op.moe_q4w_run(0, x, i_dev, w_dev, out, stream=torch.cuda.current_stream().cuda_stream)
    i_dev.copy_(torch.from_numpy(ids[:T]))
    graph.replay()
    torch.cuda.synchronize()
    assert np.array_equal(bits(bf16_out_to_f32(torch, out)), bits(outs[0][0]))
    del graph
    if fmt == "i4r":
        sel = np.arange(0, T, 97)
        assert_output_close(outs[0][0][sel], i4r.moe_forward(E, d, mid, L, synth.bf16_bits_to_f32(xb[sel]), ids[sel], w[sel], k), fmt)
    op.close()


def tc_op(torch, E, k, d, mid, max_tokens, i4r_layer):
    """A layer whose calls of every length run on the tensor cores: rotated experts, or q4cp with GEMM_TC."""
    if i4r_layer is not None:
        return make_i4r_op(torch, E, k, d, mid, max_tokens, i4r_layer)
    spec = synth.LayerSpec(experts=E, topk=k, d=d, mid=mid)
    return make_op(torch, spec, max_tokens, impl=pkg.GEMM_TC, layer=synth.make_layer(spec, seed=85))


# experts with 72, 112 and 256 rows in narrow calls, 256 in a wide one (16 * 16 > 12 * 16)
@pytest.mark.parametrize("rotated", [True, False])
@pytest.mark.parametrize("E,k,T,idle", [(64, 8, 16, 9), (64, 16, 8, 7), (64, 16, 16, 16), (16, 16, 16, 16)])
def test_repeated_ids_in_a_short_call(cuda, E, k, T, idle, rotated):
    """A padded batch of at most 16 tokens whose idle rows carry one id in every slot: that expert has more
    rows than a tile. Against the oracle (rotated layers), and bit for bit against the same tokens in a longer
    call, whose routing is another kernel's."""
    torch = cuda
    d, mid, L = 512, 256, synth.make_i4r_layer(E, 512, 256, seed=85) if rotated else None
    gen = synth.rng_for(85, T)
    ids = np.zeros((40, 16), np.int32)
    for t in range(40):
        ids[t, :k] = gen.permutation(E)[:k]
    ids[T - idle:T, :k] = 3
    w = gen.uniform(0.2, 1.0, size=(40, 16)).astype(np.float32) / k
    xb = synth.make_x(synth.rng_for(85, 9), 40, d)
    op = tc_op(torch, E, k, d, mid, 40, L)

    def run_ids(n):
        out = torch.full((n, d), float("nan"), dtype=torch.bfloat16, device="cuda")
        op.moe_q4w_run(0, bf16_tensor(torch, xb[:n], (n, d)), torch.from_numpy(ids[:n]).cuda(), torch.from_numpy(w[:n]).cuda(), out)
        op.synchronize()
        return bf16_out_to_f32(torch, out)

    y = run_ids(T)
    assert np.array_equal(bits(y), bits(run_ids(40)[:T]))
    if rotated:
        assert_output_close(y, i4r.moe_forward(E, d, mid, L, synth.bf16_bits_to_f32(xb[:T]), ids, w, k), "repeated ids T=%d" % T)
    op.close()


@pytest.mark.parametrize("rotated", [True, False])
@pytest.mark.parametrize("E,k,T,bad", [(64, 8, 16, 11), (64, 16, 16, 11), (64, 16, 8, 7), (16, 16, 16, 15)])
def test_many_non_finite_rows_in_a_short_call(cuda, E, k, T, bad, rotated):
    """A token with NaN logits takes one id k times: with many of them that expert has more rows than a tile.
    They are NaN, and the other tokens' bytes are what they are without them."""
    torch = cuda
    d, mid = 512, 256
    op = tc_op(torch, E, k, d, mid, T, synth.make_i4r_layer(E, d, mid, seed=86) if rotated else None)
    logits = synth.make_logits(synth.rng_for(86, T), T, E)
    xb = synth.make_x(synth.rng_for(86, 9), T, d)
    clean = run_i4r(torch, op, d, xb, logits)
    logits[:bad - 1] = np.nan
    logits[bad - 1] = -np.inf
    y = run_i4r(torch, op, d, xb, logits)
    assert np.isnan(y[:bad]).all() and np.isfinite(y[bad:]).all()
    assert np.array_equal(bits(y[bad:]), bits(clean[bad:]))
    op.close()


def random_blob(torch, rows, cols, fmt, seed):
    """Random codes on the GPU: q4cp with a linear code book (fmt None), or GGUF blocks, whose weights have mean zero (hidden values
    stay in the fp16 range)."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if fmt is None:
        stride = ((cols // 32 * 2) + 15) & ~15
        book = torch.linspace(-1.0, 1.0, 16, device="cuda").view(torch.uint8)
        codes = torch.randint(0, 256, (rows * cols // 2,), dtype=torch.uint8, device="cuda", generator=gen)
        scales = torch.empty(rows * stride // 2, device="cuda").uniform_(0.005, 0.03, generator=gen).half().view(torch.uint8)
        return torch.cat([book, codes, scales])
    per, n, heads = {pkg.GGML_Q5_K: (256, 176, (1e-5, 1.55e-4)), pkg.GGML_Q5_1: (32, 24, (1e-3, -1.55e-2)), pkg.GGML_Q8_0: (32, 34, (2e-4,))}[fmt]
    b = torch.randint(0, 256, (rows * cols // per, n), dtype=torch.uint8, device="cuda", generator=gen)
    for i, h in enumerate(heads):
        b[:, 2 * i:2 * i + 2] = torch.full((len(b), 1), h, device="cuda").half().view(torch.uint8)
    return b.reshape(-1)


def rows_agree(torch, E, k, d, mid, types, T, counts, extra=None):
    """A call's rows, bit for bit those of calls of 17 tokens, and the fp32 kernels' results within the roundings' bound. extra:
    (n, m): the call makes m more launches than one of its first n tokens."""
    ids = torch.from_numpy(ids_of_counts(E, k, T, counts)).cuda()
    w = torch.from_numpy(synth.rng_for(88, 1).uniform(0.2, 1.0, size=(T, 16)).astype(np.float32) / k).cuda()
    x = bf16_tensor(torch, synth.make_x(synth.rng_for(88, 9), T, d), (T, d))
    gu, dn = types

    def make(impl):
        op = pkg.MoeOperator(E, k, d, mid, T, gemm_impl=impl)
        if gu is None:
            op.load_q4cp(0, random_blob(torch, E * 2 * mid, d, gu, 1), random_blob(torch, E * d, mid, dn, 2))
        else:
            op.load_gguf(0, random_blob(torch, E * mid, d, gu, 1), random_blob(torch, E * mid, d, gu, 3), random_blob(torch, E * d, mid, dn, 2),
                         type_gu=gu, type_dn=dn)
        return op

    def run(op, t0, n):
        out = torch.full((n, d), float("nan"), dtype=torch.bfloat16, device="cuda")
        op.moe_q4w_run(0, x[t0:t0 + n].contiguous(), ids[t0:t0 + n].contiguous(), w[t0:t0 + n].contiguous(), out)
        op.synchronize()
        return out

    tc, simt = make(pkg.GEMM_TC), make(pkg.GEMM_SIMT)
    for _ in range(2):
        before = tc.launches
        whole = run(tc, 0, T)
        launches = tc.launches - before
        assert np.array_equal(np.diff(tc.get_routing(T)[4])[:len(counts)], counts)
        assert torch.isfinite(whole.float()).all()
        for t0 in (0, 17, T // 2, T - 17):
            assert torch.equal(whole[t0:t0 + 17], run(tc, t0, 17)), t0
        if extra is not None:
            before = tc.launches
            assert torch.equal(run(tc, 0, extra[0]), whole[:extra[0]])
            assert launches - (tc.launches - before) == extra[1]
    # 2-norm: both sides round to bf16 (a uniform error of 2^-9 at most: 2^-9 / sqrt(3) rms each), the tensor cores also gate, up and down
    # weights and the hidden values to fp16 (2^-11 / sqrt(3) each): sqrt(2 * 2^-18 + 4 * 2^-22) / sqrt(3) = 1.7e-3; twice that
    want = run(simt, 0, T).float()
    assert (whole.float() - want).norm() <= 3.4e-3 * want.norm()
    tc.close()
    simt.close()


# K blocks of gate/up and down with all remainders of a quad; rows on both sides of a box of 16, 32 and 48, of one and two tiles
# and of a wide tile; layers on both sides of the line for two lists
@pytest.mark.parametrize("E,k,d,mid,types", [(96, 4, 2304, 2432, (None, None)), (384, 2, 1408, 1024, (pkg.GGML_Q8_0, pkg.GGML_Q8_0)),
                                             (32, 4, 768, 320, (pkg.GGML_Q5_K, pkg.GGML_Q5_1)), (28, 4, 1152, 448, (None, None))])
def test_more_than_twelve_rows(cuda, E, k, d, mid, types):
    """Calls of more than 12 rows per expert: large layers run both forms, small ones tiles of 64 rows."""
    counts = [193, 192, 130, 129, 128, 65, 64, 63, 49, 48, 33, 32, 31, 17, 16, 15, 1]
    rows_agree(cuda, E, k, d, mid, types, max(13 * E // k + 1, 320), counts)


def popular_calls(E, k, d, mid, T):
    """A call of T tokens has the popular experts' launches, with room to the line; one of `line` tokens, where no expert can have
    enough rows, has not, and is otherwise made of the same launches."""
    least = 3 * line("kDenseGroup")
    assert T > least and T * k * d * mid > 1.5 * line("kPopularWork")
    assert form(E, k, d, mid, T) == form(E, k, d, mid, least - 1) != "few"
    return least - 1


# one group of rows more or less than the line, a whole number of them and not; two places for three popular experts (12800 rows, mid
# 6144); an odd number of K blocks; a layer of two lists
@pytest.mark.parametrize("E,k,d,mid,types", [(16, 4, 2560, 2560, (None, None)), (16, 4, 1280, 6144, (None, None)), (16, 4, 2560, 2560, (pkg.GGML_Q5_K, pkg.GGML_Q5_1)),
                                             (16, 4, 4096, 1600, (None, None)), (64, 4, 3072, 3072, (None, None))])
def test_popular_experts(cuda, E, k, d, mid, types):
    """Experts of 2304 rows and more: the down GEMM on expanded weights (two launches)."""
    n = popular_calls(E, k, d, mid, 3200)
    rows_agree(cuda, E, k, d, mid, types, 3200, [3200, 2304, 2303, 3071, 769], (n, 2))


# one list and two
@pytest.mark.parametrize("E,d,mid", [(16, 2560, 2560), (64, 3072, 3072)])
def test_popular_experts_beside_a_shared_one(cuda, E, d, mid):
    """The longest row of launches beside one another (popular experts, few rows, shared expert, wide tiles), stored and added into a residual state."""
    torch = cuda
    k, T = 4, 3200
    n = popular_calls(E, k, d, mid, T)
    counts = [3200, 2304, 2303, 3071, 769]
    ids = ids_of_counts(E, k, T, counts)
    lg = np.zeros((T, E), np.float32)
    np.put_along_axis(lg, ids[:, :k].astype(np.int64), 8.0 + 0.25 * np.arange(k, dtype=np.float32), axis=1)
    lg = torch.from_numpy(lg).cuda()
    x = bf16_tensor(torch, synth.make_x(synth.rng_for(89, 9), T, d), (T, d))
    gate_w = (torch.randn(d, device="cuda") * 0.02).bfloat16()
    blobs = [random_blob(torch, r, c, None, i) for i, (r, c) in enumerate([(E * 2 * mid, d), (E * d, mid), (mid, d), (mid, d), (d, mid)])]

    def make(impl):
        op = pkg.MoeOperator(E, k, d, mid, T, has_shared=True, gemm_impl=impl)
        op.load_q4cp(0, *blobs[:2])
        op.load_shared_q4cp(0, *blobs[2:], gate_w)
        return op

    def run(op, t0, m):
        before = op.launches
        out = torch.full((m, d), float("nan"), dtype=torch.bfloat16, device="cuda")
        op.moe_b(0, x[t0:t0 + m].contiguous(), lg[t0:t0 + m].contiguous(), out)
        op.synchronize()
        return out, op.launches - before

    tc, simt = make(pkg.GEMM_TC), make(pkg.GEMM_SIMT)
    whole, launches = run(tc, 0, T)
    assert np.array_equal(np.diff(tc.get_routing(T)[4])[:5], counts) and torch.isfinite(whole.float()).all()
    part, fewer = run(tc, 0, n)
    assert torch.equal(part, whole[:n]) and launches == fewer + 2
    for t0 in (0, 1600, T - 17):
        assert torch.equal(run(tc, t0, 17)[0], whole[t0:t0 + 17]), t0
    want = run(simt, 0, T)[0].float()
    assert (whole.float() - want).norm() <= 3.4e-3 * want.norm()   # (rows_agree's bound)
    state = torch.zeros((T, 4, d), dtype=torch.bfloat16, device="cuda")
    tc.moe_b_hc(0, x, lg, torch.zeros((T, 4), device="cuda"), state)     # gates of 2 * sigmoid(0) = 1
    tc.synchronize()
    assert torch.equal(state, whole[:, None].expand(T, 4, d))
    tc.close()
    simt.close()


def test_popular_experts_captured(cuda):
    """A captured call from hidden states (the router GEMM's clusters) with popular experts (pairs of SMs): replayed on other tokens."""
    torch = cuda
    E, k, d, mid, T = 16, 4, 2560, 2560, 3200
    n = popular_calls(E, k, d, mid, T)
    op = pkg.MoeOperator(E, k, d, mid, T)
    op.load_q4cp(0, random_blob(torch, E * 2 * mid, d, None, 1), random_blob(torch, E * d, mid, None, 2))
    gen = torch.Generator(device="cuda").manual_seed(3)
    w = torch.randn(E, d, device="cuda", generator=gen) * 0.02
    mean = torch.randn(d, device="cuda", generator=gen)
    w[[2, 5, 11]] += 0.01 * mean  # these experts' logits are the largest for most tokens
    op.load_router(0, w.bfloat16())
    tokens = [(mean + torch.randn(T, d, device="cuda", generator=gen)).bfloat16() for _ in range(2)]
    want = []
    for x in tokens:
        out = torch.full((T, d), float("nan"), dtype=torch.bfloat16, device="cuda")
        before = op.launches
        op.moe_hidden(0, x, out)
        op.synchronize()
        launches = op.launches - before
        assert np.diff(op.get_routing(T)[4]).max() >= 2304
        before = op.launches
        op.moe_hidden(0, x[:n].contiguous(), torch.empty_like(out[:n]))
        assert launches == op.launches - before + 2
        want.append(out)
    assert all(torch.isfinite(y.float()).all() for y in want) and not torch.equal(want[0], want[1])
    x, out = tokens[0].clone(), torch.empty((T, d), dtype=torch.bfloat16, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        op.moe_hidden(0, x, out, stream=torch.cuda.current_stream().cuda_stream)
    for y, z in zip(tokens, want):
        x.copy_(y)
        out.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, z)
    del graph
    op.synchronize()
    op.close()
