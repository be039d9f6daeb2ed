"""Performance cases of the routed-expert MoE layer.

A case is one call of a public entry point of `MoeOperator` on a loaded layer: shapes, weight format,
entry point, number of tokens and routing skew. The listed cases run from one decoded token to a
16384-token prefill chunk; `draw` gives further cases of the same ranges. Weights and inputs are made
on the GPU from the seed, with the value distributions of the repository's benchmark; the calls on
host buffers get theirs in pinned host memory.
"""
import math

import numpy as np
import torch

import gfx1151_engine_b200 as pkg
from gfx1151_engine_b200 import synth

# Layer shapes: the ~177B-MoE layer of the benchmark, the engine's own layer, the small parity layer.
BIG = {"experts": 512, "topk": 10, "d": 4096, "mid": 1024}
ENGINE = {"experts": 512, "topk": 10, "d": 2560, "mid": 640}
SMALL = {"experts": 64, "topk": 8, "d": 2048, "mid": 512}

# Weight formats: bytes per weight of gate/up and of down as they stand in a model file.
FORMATS = {
    "q4cp": (0.5625, 0.5625),
    "q4k_q51": (144 / 256, 24 / 32),
    "q5k_q51": (176 / 256, 24 / 32),
    "iq4xs": (136 / 256, 136 / 256),
    "q80": (34 / 32, 34 / 32),
    "i4r": (0.5 + 2 / 128, 0.5 + 2 / 128),
}
GGUF_TYPES = {"q4k_q51": (pkg.GGML_Q4_K, pkg.GGML_Q5_1), "q5k_q51": (pkg.GGML_Q5_K, pkg.GGML_Q5_1),
              "iq4xs": (pkg.GGML_IQ4_XS, pkg.GGML_IQ4_XS), "q80": (pkg.GGML_Q8_0, pkg.GGML_Q8_0)}


def _case(name, shape, T, fmt="q4cp", shared=False, entry="moe_b", skew=0.0):
    c = dict(shape, tokens=T, fmt=fmt, shared=shared, entry=entry, skew=skew)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one decoded token of one stream: latency and launches
        _case("decode_1", BIG, 1, shared=True),
        # speculative verify: four drafted tokens and the last accepted one
        _case("verify_5", BIG, 5, shared=True),
        # the same on a GGUF checkpoint
        _case("gguf_verify_5", BIG, 5, fmt="q4k_q51"),
        # a small layer whose router runs inside the operator, as many tokens as decode takes
        _case("small_hidden_16", SMALL, 16, entry="moe_hidden"),
        # decode of a batch of streams, an odd number of them
        _case("batch_13", BIG, 13, shared=True),
        # a short prompt, ragged
        _case("prompt_77", BIG, 77, shared=True, skew=0.5),
        # a prefill chunk of the engine's own layer, added into its residual state
        _case("engine_chunk_500", ENGINE, 500, shared=True, entry="moe_b_hc", skew=0.5),
        # the engine's usual prefill chunk on rotated 4-bit experts
        _case("i4r_chunk_2048", ENGINE, 2048, fmt="i4r", skew=0.5),
        # a caller with host buffers
        _case("host_chunk_4096", BIG, 4096, entry="moe_b_host", skew=1.0),
        # a long chunk of a GGUF checkpoint
        _case("gguf_chunk_8192", BIG, 8192, fmt="q4k_q51", skew=1.0),
        # the largest chunk: the benchmark's prefill call
        _case("prefill_16384", BIG, 16384, skew=1.0),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: tokens over four decades, shapes from small layers to the benchmark's, every
    format and entry point in the proportions in which they are used."""
    r = rng.random()
    if r < 0.4:
        shape = dict(BIG)
    elif r < 0.7:
        shape = dict(ENGINE)
    else:
        shape = {"experts": rng.choice([16, 60, 64, 100, 128, 256, 384]), "topk": rng.choice([2, 4, 6, 8]),
                 "d": 256 * rng.randint(4, 16), "mid": 128 * rng.randint(2, 8)}
    # a third decode and verify calls, the rest prompts and chunks
    T = rng.randint(1, 16) if rng.random() < 0.34 else _log_uniform(rng, 17, 16384)
    fmt = rng.choice(["q4cp"] * 4 + ["q4k_q51"] * 2 + ["q5k_q51", "iq4xs", "q80", "i4r"])
    if fmt == "iq4xs" and shape["mid"] % 256:
        fmt = "q4k_q51"  # those blocks hold 256 columns
    entry = rng.choice(["moe_b"] * 5 + ["moe_b_hc", "moe_q4w_run"] + ["moe_hidden"] * 2 + (["moe_b_host"] if T >= 64 else []))
    shared = fmt == "q4cp" and rng.random() < 0.6
    if fmt == "i4r" and 2 * shape["mid"] > shape["d"]:
        shape["mid"] = shape["d"] // 256 * 128
    return _case(None, shape, T, fmt=fmt, shared=shared, entry=entry, skew=rng.choice([0.0, 0.5, 1.0]) if T > 16 else 0.0)


# ------------------------------------------------------------------ weights and inputs
def _book():
    """A symmetric non-uniform 4-bit code book with largest magnitude 1 (quantiles of a normal distribution),
    the kind that q4cp checkpoints carry."""
    q = (np.arange(8) + 0.5) / 16.0 + 0.5
    t = torch.distributions.Normal(0.0, 1.0).icdf(torch.from_numpy(q)).numpy()
    t = t / t[-1]
    return np.concatenate([-t[::-1], t]).astype("<f4")


def _bytes(n, gen):
    """n random bytes."""
    out = torch.empty((n + 7) // 8, dtype=torch.int64, device="cuda").random_(generator=gen)
    out = out.view(torch.uint8)
    out[7::8] = out[6::8] ^ out[0::8]  # random_ leaves the sign bit clear
    return out[:n]


def _abs_normal(n, sigma, gen):
    out = torch.empty(n, dtype=torch.float32, device="cuda")
    return out.normal_(0.0, sigma, generator=gen).abs_()


def _f16_bytes(t, width):
    return t.half().view(torch.uint8).view(-1, 2 * width)


def _q4cp(rows, cols, gen):
    stride = ((cols // 32 * 2) + 15) & ~15
    ncode = rows * cols // 2
    out = torch.zeros(synth.q4cp_nbytes(rows, cols), dtype=torch.uint8, device="cuda")
    out[:64] = torch.from_numpy(_book().view(np.uint8).copy()).cuda()
    out[64:64 + ncode] = _bytes(ncode, gen)
    sc = _abs_normal(rows * (cols // 32), 0.02, gen)
    out[64 + ncode:].view(rows, stride)[:, :cols // 32 * 2] = _f16_bytes(sc, 1).view(rows, -1)
    return out


def _i4r(rows, cols, gen):
    ncode = rows * cols // 2
    out = torch.empty(synth.i4r_nbytes(rows, cols), dtype=torch.uint8, device="cuda")
    out[:ncode] = _bytes(ncode, gen)
    sc = torch.empty(rows * (cols // 128), dtype=torch.float32, device="cuda").normal_(0.0, 0.02 / 8, generator=gen)
    out[ncode:] = sc.half().view(torch.uint8)
    return out


def _planes(n, gen):
    sign = torch.randint(0, 2, (n,), device="cuda", generator=gen) * 2 - 1
    return (sign * torch.empty(n, device="cuda").uniform_(0.5, 1.5, generator=gen)).half()


def _gguf(rows, cols, gtype, gen):
    """Raw GGUF blocks with uniform codes and block scales that keep |w| <= |N(0, 0.02)|."""
    per, size = {pkg.GGML_Q4_K: (256, 144), pkg.GGML_Q5_K: (256, 176), pkg.GGML_Q5_1: (32, 24),
                 pkg.GGML_IQ4_XS: (256, 136), pkg.GGML_Q8_0: (32, 34)}[gtype]
    nb = rows * (cols // per)
    out = _bytes(nb * size, gen).view(nb, size)
    a = _abs_normal(nb, 0.02, gen)
    if gtype == pkg.GGML_Q4_K:
        heads = [a / (63.0 * 15.0), a / (63.0 * 2.0)]
    elif gtype == pkg.GGML_Q5_K:
        heads = [a / (63.0 * 31.0), a / (63.0 * 2.0)]
    elif gtype == pkg.GGML_Q5_1:
        heads = [a / 31.0, -a / 2.0]
    elif gtype == pkg.GGML_IQ4_XS:
        heads = [a / (32.0 * 127.0)]
    else:
        heads = [a / 127.0]
    for i, h in enumerate(heads):
        out[:, 2 * i:2 * i + 2] = _f16_bytes(h, 1)
    return out.view(-1)


def _draw_inputs(case, seed):
    """The raw weights and inputs of a case, on the GPU, from the seed alone."""
    E, d, mid, T = case["experts"], case["d"], case["mid"], case["tokens"]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    raw = {}
    if case["fmt"] == "q4cp":
        raw["gate_up"], raw["down"] = _q4cp(E * 2 * mid, d, gen), _q4cp(E * d, mid, gen)
    elif case["fmt"] == "i4r":
        raw["gate_up"], raw["down"] = _i4r(E * 2 * mid, d, gen), _i4r(E * d, mid, gen)
        raw["planes"] = _planes(d, gen), _planes(2 * mid, gen), _planes(mid, gen), _planes(d, gen)
    else:
        gu, dn = GGUF_TYPES[case["fmt"]]
        raw["gate"], raw["up"], raw["down"] = _gguf(E * mid, d, gu, gen), _gguf(E * mid, d, gu, gen), _gguf(E * d, mid, dn, gen)
    if case["shared"]:
        raw["sh_gate_w"] = torch.empty(d, device="cuda").normal_(0.0, 0.02, generator=gen).bfloat16()
        raw["shared"] = _q4cp(mid, d, gen), _q4cp(mid, d, gen), _q4cp(d, mid, gen)
    raw["x"] = torch.empty(T, d, device="cuda").normal_(0.0, 1.0, generator=gen).bfloat16()
    raw["logits"] = torch.empty(T, E, device="cuda").normal_(0.0, 1.0, generator=gen)
    if case["skew"]:
        raw["logits"] += torch.from_numpy(synth.zipf_bias(synth.rng_for(seed, 77), E, strength=case["skew"])).cuda()
    if case["entry"] == "moe_hidden":
        raw["router"] = torch.empty(E, d, device="cuda").normal_(0.0, 0.02, generator=gen).bfloat16()
    elif case["entry"] == "moe_b_hc":
        raw["w4"] = torch.empty(T, 4, device="cuda").normal_(0.0, 2.0, generator=gen)
        raw["residual"] = torch.empty(T, 4, d, device="cuda").normal_(0.0, 1.0, generator=gen).bfloat16()
    return raw


def prepare(case, seed):
    E, k, d, mid, T = case["experts"], case["topk"], case["d"], case["mid"], case["tokens"]
    raw = _draw_inputs(case, seed)
    op = pkg.MoeOperator(E, k, d, mid, max(T, 16), has_shared=case["shared"])
    if case["fmt"] == "q4cp":
        op.load_q4cp(0, raw["gate_up"], raw["down"])
    elif case["fmt"] == "i4r":
        op.load_i4r(0, raw["gate_up"], raw["down"], *raw["planes"])
    else:
        gu, dn = GGUF_TYPES[case["fmt"]]
        op.load_gguf(0, raw["gate"], raw["up"], raw["down"], type_gu=gu, type_dn=dn)
    if case["shared"]:
        op.load_shared_q4cp(0, *raw["shared"], raw["sh_gate_w"])
    x, logits = raw["x"], raw["logits"]
    state = {"case": case, "op": op, "x": x, "logits": logits, "out": torch.empty(T, d, dtype=torch.bfloat16, device="cuda")}
    entry = case["entry"]
    if entry == "moe_hidden":
        op.load_router(0, raw["router"])
    elif entry == "moe_b_hc":
        state["w4"], state["residual"] = raw["w4"], raw["residual"]
    elif entry == "moe_q4w_run":
        state["ids"] = torch.zeros(T, 16, dtype=torch.int32, device="cuda")
        state["w"] = torch.zeros(T, 16, device="cuda")
        op.router_topk_b(logits, state["ids"], state["w"])
    elif entry == "moe_b_host":
        for n in ("x", "logits", "out"):
            state[n] = state[n].cpu().pin_memory()
    torch.cuda.synchronize()
    del raw
    torch.cuda.empty_cache()  # the source tensors may be freed once they are loaded
    return state


def run(state):
    op, entry, x, out = state["op"], state["case"]["entry"], state["x"], state["out"]
    if entry == "moe_b":
        op.moe_b(0, x, state["logits"], out)
    elif entry == "moe_hidden":
        op.moe_hidden(0, x, out)
    elif entry == "moe_b_hc":
        op.moe_b_hc(0, x, state["logits"], state["w4"], state["residual"])
        return state["residual"]
    elif entry == "moe_q4w_run":
        op.moe_q4w_run(0, x, state["ids"], state["w"], out)
    else:
        op.moe_b_host(0, x, state["logits"], out, state["case"]["tokens"])
    return out


def _experts_used(case):
    """Number of distinct experts that a call's tokens choose (one simulated routing; weights of the others are not read)."""
    E, k, T = case["experts"], case["topk"], case["tokens"]
    rng = synth.rng_for(1, T)
    bias = synth.zipf_bias(synth.rng_for(1, 77), E, strength=case["skew"])
    used = np.zeros(E, bool)
    for t0 in range(0, T, 2048):
        lg = rng.normal(0.0, 1.0, size=(min(2048, T - t0), E)).astype(np.float32) + bias
        used[np.argpartition(-lg, k - 1, axis=1)[:, :k].reshape(-1)] = True
    return int(used.sum())


def work(case):
    E, k, d, mid, T = case["experts"], case["topk"], case["d"], case["mid"], case["tokens"]
    gu, dn = FORMATS[case["fmt"]]
    per_expert = 2 * mid * d * gu + d * mid * dn
    nbytes = _experts_used(case) * per_expert + T * d * 2
    pairs = T * k
    if case["shared"]:
        nbytes += 3 * mid * d * 0.5625 + d * 2
        pairs += T
    if case["entry"] == "moe_hidden":
        nbytes += E * d * 2
    elif case["entry"] == "moe_q4w_run":
        nbytes += T * k * 8
    else:
        nbytes += T * E * 4
    nbytes += T * d * 2 * (8 if case["entry"] == "moe_b_hc" else 1)  # the residual state is read and written
    flops = 6.0 * pairs * d * mid + (2.0 * T * E * d if case["entry"] == "moe_hidden" else 0.0)
    return {"bytes": float(nbytes), "flops": flops}


def tolerance(case):
    """fp16 operands, fp32 sums, a bf16 result. Against the fp32 kernels on the same inputs the calls above differ by
    1.5e-3 in the 2-norm and by one bf16 step (7.8e-3) at most; the residual write-back, which adds the result to a
    state of norm 1 before it rounds, by 2.4e-4. Four times that is stated."""
    return {"rel": 1e-3 if case["entry"] == "moe_b_hc" else 6e-3, "max": 0.032}


# ------------------------------------------------------------------ the same in 64 bits
def _f16_at(blocks, byte):
    return blocks[:, byte:byte + 2].contiguous().view(torch.float16).double()


def _nibbles(codes):
    """Low nibbles, then high nibbles: [n][bytes] -> [n][2][bytes]."""
    return torch.stack([codes & 15, codes >> 4], 1)


def _q4cp_rows(blob, rows, cols, r0, n):
    """Rows r0 .. r0+n-1; byte i of a row holds columns 2i and 2i+1."""
    stride = ((cols // 32 * 2) + 15) & ~15
    codes = blob[64 + r0 * cols // 2:64 + (r0 + n) * cols // 2].view(n, -1)
    book = blob[:64].view(torch.float32).double()
    off = 64 + rows * cols // 2
    sc = blob[off + r0 * stride:off + (r0 + n) * stride].view(n, stride)[:, :cols // 32 * 2].contiguous().view(torch.float16).double()
    return book[_nibbles(codes).transpose(1, 2).reshape(n, cols).long()] * sc.repeat_interleave(32, 1)


def _i4r_rows(blob, rows, cols, r0, n):
    codes = blob[r0 * cols // 2:(r0 + n) * cols // 2].view(n, -1)
    off, per = rows * cols // 2, cols // 128
    sc = blob[off + r0 * per * 2:off + (r0 + n) * per * 2].view(torch.float16).view(n, per).double()
    return (_nibbles(codes).transpose(1, 2).reshape(n, cols).double() - 8.0) * sc.repeat_interleave(128, 1)


_GRID = (-127, -104, -83, -65, -49, -35, -22, -10, 1, 13, 25, 38, 53, 69, 89, 113)


def _gguf_rows(blob, cols, gtype, r0, n):
    per, size = {pkg.GGML_Q4_K: (256, 144), pkg.GGML_Q5_K: (256, 176), pkg.GGML_Q5_1: (32, 24),
                 pkg.GGML_IQ4_XS: (256, 136), pkg.GGML_Q8_0: (32, 34)}[gtype]
    b = blob.view(-1, size)[r0 * (cols // per):(r0 + n) * (cols // per)]
    nb = b.shape[0]
    if gtype == pkg.GGML_Q8_0:
        w = _f16_at(b, 0) * b[:, 2:].contiguous().view(torch.int8).double()
    elif gtype == pkg.GGML_Q5_1:
        bits = torch.stack([b[:, 4 + j // 8] >> (j % 8) & 1 for j in range(32)], 1)
        w = _f16_at(b, 0) * (_nibbles(b[:, 8:]).reshape(nb, 32) + 16 * bits).double() + _f16_at(b, 2)
    elif gtype == pkg.GGML_IQ4_XS:
        low = torch.stack([b[:, 4 + i // 2] >> (4 * (i % 2)) & 15 for i in range(8)], 1)
        high = torch.stack([b[:, 2 + i // 4] >> (2 * (i % 4)) & 3 for i in range(8)], 1)
        sc = _f16_at(b, 0) * ((low | high << 4).double() - 32.0)
        grid = torch.tensor(_GRID, dtype=torch.float64, device=b.device)
        w = sc[:, :, None] * grid[_nibbles(b[:, 8:].reshape(nb * 8, 16)).reshape(nb, 8, 32).long()]
    else:
        p = b[:, 4:16].int()
        sc = torch.cat([p[:, 0:4] & 63, (p[:, 8:12] & 15) | (p[:, 0:4] >> 6 << 4)], 1).double() * _f16_at(b, 0)
        mn = torch.cat([p[:, 4:8] & 63, (p[:, 8:12] >> 4) | (p[:, 4:8] >> 6 << 4)], 1).double() * _f16_at(b, 2)
        q = _nibbles(b[:, -128:].reshape(nb * 4, 32)).reshape(nb, 8, 32).int()
        if gtype == pkg.GGML_Q5_K:
            q = q + 16 * torch.stack([b[:, 16:48] >> i & 1 for i in range(8)], 1)
        w = sc[:, :, None] * q.double() - mn[:, :, None]
    return w.reshape(n, cols)


def _hadamard(v):
    """128-point orthonormal Hadamard transform of every block of the last axis."""
    h = torch.ones(1, 1, dtype=torch.float64, device=v.device)
    for _ in range(7):
        h = torch.cat([torch.cat([h, h], 1), torch.cat([h, -h], 1)], 0)
    return (v.reshape(-1, 128) @ h).reshape(v.shape) / math.sqrt(128.0)


def exact(case, seed):
    """The layer in 64 bits: softmax, top-k, renormalised weights, SwiGLU experts, shared expert behind its sigmoid gate."""
    E, k, d, mid, fmt = case["experts"], case["topk"], case["d"], case["mid"], case["fmt"]
    raw = _draw_inputs(case, seed)
    x = raw["x"].double()
    logits = x @ raw["router"].double().T if case["entry"] == "moe_hidden" else raw["logits"].double()
    w, ids = torch.topk(torch.softmax(logits, 1), k, dim=1)
    w = w / w.sum(1, keepdim=True)
    xin = x
    if fmt == "i4r":
        pre_gu, post_gu, pre_dn, post_dn = [p.double() for p in raw["planes"]]
        xin = _hadamard(x * pre_gu)
    y = torch.zeros_like(x)
    silu = torch.nn.functional.silu
    for e in range(E):
        tok, slot = torch.nonzero(ids == e, as_tuple=True)
        if not len(tok):
            continue
        if fmt in ("q4cp", "i4r"):
            rows = _q4cp_rows if fmt == "q4cp" else _i4r_rows
            gu = rows(raw["gate_up"], E * 2 * mid, d, e * 2 * mid, 2 * mid)
            dn = rows(raw["down"], E * d, mid, e * d, d)
        else:
            tg, td = GGUF_TYPES[fmt]
            gu = torch.cat([_gguf_rows(raw[n], d, tg, e * mid, mid) for n in ("gate", "up")])
            dn = _gguf_rows(raw["down"], mid, td, e * d, d)
        z = xin[tok] @ gu.T
        if fmt == "i4r":
            z = _hadamard(z) * post_gu
        h = silu(z[:, :mid]) * z[:, mid:]
        if fmt == "i4r":
            h = _hadamard(h * pre_dn)
        y.index_add_(0, tok, (h @ dn.T) * w[tok, slot, None])
    if fmt == "i4r":
        y = _hadamard(y) * post_dn
    if case["shared"]:
        g, u, dn = raw["shared"]
        h = silu(x @ _q4cp_rows(g, mid, d, 0, mid).T) * (x @ _q4cp_rows(u, mid, d, 0, mid).T)
        y += torch.sigmoid(x @ raw["sh_gate_w"].double())[:, None] * (h @ _q4cp_rows(dn, d, mid, 0, d).T)
    if case["entry"] == "moe_b_hc":
        return raw["residual"].double() + 2.0 * torch.sigmoid(raw["w4"].double() / 4.0)[:, :, None] * y[:, None, :]
    return y
