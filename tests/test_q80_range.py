"""Q8_0 layers on the fp32 kernels: activations and hidden values so large that code * value leaves the fp32 range where
scale * code * value does not, in all numbers of rows that the kernels know, against 64 bits."""
import numpy as np
import pytest

import gfx1151_engine_b200 as pkg
from gfx1151_engine_b200 import synth
from helpers import bf16_out_to_f32, bf16_tensor

pytestmark = pytest.mark.gpu


def blocks(scales, codes):
    """[rows][blocks] scales and [rows][blocks][32] int8 codes as raw Q8_0 blocks."""
    return np.concatenate([scales.astype("<f2")[..., None].view(np.uint8), codes.astype(np.int8).view(np.uint8)], axis=-1).reshape(-1)


# the decode kernels of a layer that the GEMV does not take (d > 2048), and the cross-check
@pytest.mark.parametrize("impl,d", [(pkg.GEMM_AUTO, 2304), (pkg.GEMM_SIMT, 256)])
def test_large_values(cuda, impl, d):
    torch = cuda
    E, mid, T = 2, 64, 13
    gen = np.random.default_rng(7)
    raw, w = [], []
    for rows, cols in ((E * mid, d), (E * mid, d), (E * d, mid)):
        sc, q = np.zeros((rows, cols // 32), np.float32), np.zeros((rows, cols // 32, 32), np.int64)
        if len(raw) == 0:                       # gate: columns 0..31, whose activations are about 1e36
            sc[:, 0], q[:, 0] = 2.0 ** -10, gen.integers(100, 128, size=(rows, 32))
        elif len(raw) == 1:                     # up: the other columns, with sums of about 1
            sc[:, 1:], q[:, 1:] = 2.0 ** -8, gen.integers(4, 13, size=(rows, cols // 32 - 1, 32))
        else:
            sc[:], q[:] = 2.0 ** -20, gen.integers(-127, 128, size=q.shape)
        raw.append(torch.from_numpy(blocks(sc, q)).cuda())
        w.append((sc[..., None].astype(np.float64) * q).reshape(rows, cols))
    x = gen.uniform(0.5, 1.5, size=(T, d))
    x[:, :32] *= 1e36
    x[:, 64:] *= 0.01
    xb = synth.f32_to_bf16_bits(x.astype(np.float32))
    x = synth.bf16_bits_to_f32(xb).astype(np.float64)
    op = pkg.MoeOperator(E, 1, d, mid, 16, gemm_impl=impl)
    op.load_gguf(0, *raw, type_gu=pkg.GGML_Q8_0, type_dn=pkg.GGML_Q8_0)
    for rows in (1, 2, 3, 8, 9):                # of expert 0; the other tokens take expert 1
        ids = np.zeros((T, 16), np.int32)
        ids[rows:, 0] = 1
        out = torch.full((T, d), float("nan"), dtype=torch.bfloat16, device="cuda")
        op.moe_q4w_run(0, bf16_tensor(torch, xb, (T, d)), torch.from_numpy(ids).cuda(), torch.ones(T, 16, device="cuda"), out)
        op.synchronize()
        y = bf16_out_to_f32(torch, out)
        for t in range(T):
            e = ids[t, 0]
            h = (w[0][e * mid:(e + 1) * mid] @ x[t]) * (w[1][e * mid:(e + 1) * mid] @ x[t])      # silu(g) = g: g is about 4e36
            terms = w[2][e * d:(e + 1) * d] * h
            assert 127 * np.abs(h).max() > 3.4e38 and 100 * 32 * 1e36 * 0.5 > 3.4e38
            # bf16 rounding, and fp32 roundings of every sum (at most (2 * d + mid) of 2^-24 of its terms)
            assert (np.abs(y[t] - terms.sum(1)) <= 2.0 ** -8 * np.abs(terms.sum(1)) + (2 * d + mid) * 2.0 ** -24 * np.abs(terms).sum(1)).all(), (rows, t)
    op.close()
