"""GPU: products of a few activation rows (csrc/gemm_few.cu) against the oracle, at the edges of its
tiles: 128 weight rows, 8 activation rows, units of 256 k dealt out in runs that cross tiles.

Tolerances: both f16 operands are rounded once, 2^-11 of each value, so the error of a sum of K products of
independent sign is about 2^-11 of its root mean square (max over the results: 1e-3 of the largest
one). Block sums of the int8 form are exact: only the order of f32 additions differs, 1e-5.
"""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

SHAPES = [(2, 128, 256), (8, 131, 512), (9, 40, 2816), (16, 1000, 768), (17, 520, 1024),
          (25, 4099, 512), (33, 257, 256), (48, 300, 1280), (49, 127, 2048), (64, 2056, 768)]


def run(ctx, kb, torch, dt, blocks, x, N, act, shift=0):
    """`shift` floats in front of x: rows that start on no 16-byte boundary."""
    M, K = x.shape
    buf = torch.zeros(M * K + 4, dtype=torch.float32, device="cuda")
    buf[shift:shift + M * K] = torch.from_numpy(x.reshape(-1)).cuda()
    y = torch.full((M, N), float("nan"), dtype=torch.float32, device="cuda")
    fn = ctx.gemm_q8_0 if dt == kb.DTYPE_Q8_0 else ctx.gemm_q4_k
    w = torch.from_numpy(np.ascontiguousarray(blocks)).cuda()
    torch.cuda.synchronize()
    fn(w, buf[shift:shift + M * K], y, M, N, K, act)
    ctx.sync()
    return y.cpu().numpy()


def data(M, N, K):
    rng = np.random.Generator(np.random.PCG64(0xB2000C00 + M * 7 + N * 3 + K))
    return ((rng.standard_normal((N, K)) * 0.02).astype(np.float32),
            rng.standard_normal((M, K)).astype(np.float32))


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("fmt", ["q8_0", "q4_k"])
def test_few_rows(ctx, kb, oracle, torch_cuda, fmt, M, N, K, shift):
    if fmt == "q4_k" and M < 9:
        pytest.skip("the GEMV's, which asks for 16-byte aligned activations")
    w, x = data(M, N, K)
    if fmt == "q8_0":
        blocks, dt = oracle.quantize_weights_q8_0(w), kb.DTYPE_Q8_0
        ref = oracle.gemm_q8_0(blocks, x, M, N, K)
    else:
        blocks, dt = oracle.quantize_weights_q4_k(w), kb.DTYPE_Q4_K
        ref = oracle.gemm_q4_k(blocks, x, M, N, K)
    assert rel_err(run(ctx, kb, torch_cuda, dt, blocks, x, N, kb.ACT_F32, shift), ref) <= 1e-3


@pytest.mark.parametrize("M,N,K", SHAPES[2:] + [(65, 300, 512), (100, 129, 1024), (137, 200, 256)])
def test_few_rows_q8_activations(ctx, kb, oracle, torch_cuda, M, N, K):
    w, x = data(M, N, K)
    x[M // 2, :32] = 0  # a block of zeros has the scale 0
    blocks = oracle.quantize_weights_q8_0(w)
    ref = oracle.gemm_q8_0(blocks, x, M, N, K, oracle.ACT_Q8)
    for shift in (0, 3):
        got = run(ctx, kb, torch_cuda, kb.DTYPE_Q8_0, blocks, x, N, kb.ACT_Q8, shift)
        assert rel_err(got, ref) <= 1e-5
