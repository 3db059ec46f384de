"""GPU: products of a few activation rows (csrc/gemm_few.cu) against the oracle, at the edges of its
tiles: 128 weight rows (int8: 112 or 128), 8 activation rows, units of 256 k, one a CTA and in runs that
cross tiles.

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


def matrix(fmt, N, K):
    """Random blocks [N x K] of ordinary size, and their bytes per row."""
    rng = np.random.Generator(np.random.PCG64(0xB2000C80 + N + K))
    if fmt == "q8_0":
        b = rng.integers(0, 256, (N, K // 32, 34), dtype=np.uint8)
        b[..., :2] = (rng.uniform(0.5, 2, (N, K // 32, 1)) * 1e-4).astype(np.float16).view(np.uint8)
    else:
        b = rng.integers(0, 256, (N, K // 256, 144), dtype=np.uint8)
        b[..., :2] = (rng.uniform(0.5, 2, (N, K // 256, 1)) * 1e-4).astype(np.float16).view(np.uint8)
        b[..., 2:4] = (rng.uniform(3, 12, (N, K // 256, 1)) * 1e-4).astype(np.float16).view(np.uint8)
    return b.reshape(N, -1)


def some_rows(N):
    edges = [0, 1, 111, 112, 127, 128, N - 129, N - 113, N - 2, N - 1]
    return np.unique(edges + list(range(5, N, N // 40)))


def several_calls(ctx, kb, torch, fmt, blocks, x, N, act, calls=4):
    """The result of every one of `calls` calls, behind one another on the stream."""
    M, K = x.shape
    w, xd = torch.from_numpy(blocks).cuda(), torch.from_numpy(x).cuda()
    ys = [torch.full((M, N), float("nan"), dtype=torch.float32, device="cuda") for _ in range(calls)]
    torch.cuda.synchronize()
    for y in ys:
        (ctx.gemm_q8_0 if fmt == "q8_0" else ctx.gemm_q4_k)(w, xd, y, M, N, K, act)
    ctx.sync()
    return [y.cpu().numpy() for y in ys]


# 1456 units of 112 tiles over 148 or 296 CTAs: runs longer than the ring that begin and end inside
# tiles; 33 x 16 units: one to four a CTA; 2 x 16: sixteen CTAs to a tile
@pytest.mark.parametrize("N,K", [(14336, 3328), (4099, 4096), (200, 4096)])
@pytest.mark.parametrize("fmt,M", [("q8_0", m) for m in (2, 9, 17, 32, 48, 64)] +
                         [("q4_k", m) for m in (9, 24, 25, 48, 64)])
def test_runs_across_tiles(ctx, kb, oracle, torch_cuda, fmt, M, N, K):
    """Long runs give the oracle's results. Calls differ by the order in which a tile's runs are added:
    up to 16 additions of 2^-24 of the sums each, 1e-6 of the largest result."""
    blocks = matrix(fmt, N, K)
    x = data(M, 1, K)[1]
    got = several_calls(ctx, kb, torch_cuda, fmt, blocks, x, N, kb.ACT_F32)
    pick = some_rows(N)
    sub = np.ascontiguousarray(blocks[pick]).reshape(-1)
    ref = (oracle.gemm_q8_0 if fmt == "q8_0" else oracle.gemm_q4_k)(sub, x, M, pick.size, K)
    for y in got:
        assert rel_err(y[:, pick], ref) <= 1e-3
        assert rel_err(y, got[0]) <= 1e-6


# Matrices whose K stays whole: 93 tiles of 112 rows, 148 of 128, and a K of fewer than four units
@pytest.mark.parametrize("M,N,K", [(24, 10400, 2048), (48, 10400, 2048), (64, 10400, 2048),
                                   (96, 10400, 2048), (33, 18944, 2304), (128, 18944, 2304),
                                   (16, 1000, 512), (128, 300, 768), (9, 131, 256),
                                   (104, 10400, 2048), (128, 10400, 2048), (90, 18944, 2304),
                                   (112, 18944, 2304)])
def test_q8_activations_bit_exact(ctx, kb, oracle, torch_cuda, M, N, K):
    blocks = matrix("q8_0", N, K)
    x = data(M, 1, K)[1]
    got = several_calls(ctx, kb, torch_cuda, "q8_0", blocks, x, N, kb.ACT_Q8, 1)[0]
    pick = some_rows(N)
    ref = oracle.gemm_q8_0(np.ascontiguousarray(blocks[pick]).reshape(-1), x, M, pick.size, K,
                           oracle.ACT_Q8)
    assert (got[:, pick] == ref).all()


@pytest.mark.parametrize("byte", [0x80, 0x7F, 0x00])
def test_q8_activations_largest_block_sums(ctx, kb, oracle, torch_cuda, byte):
    """32 products of -128 or 127 with +-127 are the largest sums a block can have."""
    M, N, K = 12, 136, 512
    blocks = matrix("q8_0", N, K)
    blocks.reshape(N, -1, 34)[..., 2:] = byte
    x = np.ones((M, K), np.float32)
    x[1::2] = -3.0
    got = several_calls(ctx, kb, torch_cuda, "q8_0", blocks, x, N, kb.ACT_Q8, 1)[0]
    assert (got == oracle.gemm_q8_0(blocks.reshape(-1), x, M, N, K, oracle.ACT_Q8)).all()


@pytest.mark.parametrize("M,N,K", [(16, 8000, 2048), (33, 2048, 1280)])
def test_q8_activations_halved_k_repeats(ctx, kb, oracle, torch_cuda, M, N, K):
    blocks = matrix("q8_0", N, K)
    got = several_calls(ctx, kb, torch_cuda, "q8_0", blocks, data(M, 1, K)[1], N, kb.ACT_Q8)
    for again in got[1:]:
        assert (got[0] == again).all()


# K in four and eight parts of two, four and five units a CTA: 14 warps, and 28. The parts' sums are added in
# any order (1e-5, as above).
@pytest.mark.parametrize("M", [113, 128])
@pytest.mark.parametrize("N,K", [(2048, 2048), (2048, 8192), (2048, 10240)])
def test_q8_activations_in_parts(ctx, kb, oracle, torch_cuda, M, N, K):
    blocks = matrix("q8_0", N, K)
    x = data(M, 1, K)[1]
    got = several_calls(ctx, kb, torch_cuda, "q8_0", blocks, x, N, kb.ACT_Q8)[0]
    pick = np.r_[0:130, N - 40:N]
    ref = oracle.gemm_q8_0(np.ascontiguousarray(blocks[pick]).reshape(-1), x, M,
                           len(pick), K, oracle.ACT_Q8)
    assert rel_err(got[:, pick], ref) <= 1e-5


@pytest.mark.parametrize("M", [513, 530, 576, 584])
@pytest.mark.parametrize("fmt", ["q8_0", "q4_k"])
def test_rows_behind_a_pass_of_512(ctx, kb, oracle, torch_cuda, fmt, M):
    N, K = 300, 512
    w, x = data(M, N, K)
    if fmt == "q8_0":
        blocks, dt = oracle.quantize_weights_q8_0(w), kb.DTYPE_Q8_0
        ref = oracle.gemm_q8_0(blocks, x, M, N, K)
    else:
        blocks, dt = oracle.quantize_weights_q4_k(w), kb.DTYPE_Q4_K
        ref = oracle.gemm_q4_k(blocks, x, M, N, K)
    assert rel_err(run(ctx, kb, torch_cuda, dt, blocks, x, N, kb.ACT_F32), ref) <= 1e-3
