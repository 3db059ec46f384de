"""GPU: activations of the TMA-staged product (csrc/gemm_tma.cu) at the edges of what lays them out (32
rows x 256 k, a padded end of the stream), of its rings (128 | 129, 256 | 257, 512 rows) and for rows
that start on no 16-byte boundary. The oracle and the tolerance of test_gemm_few_gpu.py."""
import pytest

from conftest import rel_err
from test_gemm_few_gpu import data, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K,shift", [(65, 300, 256, 0), (97, 129, 768, 1), (128, 257, 1280, 0),
                                         (129, 128, 256, 3), (256, 70, 2816, 0), (257, 140, 768, 0),
                                         (300, 130, 1024, 2), (512, 200, 512, 0)])
@pytest.mark.parametrize("fmt", ["q8_0", "q4_k"])
def test_rows(ctx, kb, oracle, torch_cuda, fmt, M, N, K, shift):
    w, x = data(M, N, K)
    if fmt == "q8_0":
        blocks, dt = oracle.quantize_weights_q8_0(w), kb.DTYPE_Q8_0
        ref = oracle.gemm_q8_0(blocks, x, M, N, K)
    else:
        blocks, dt = oracle.quantize_weights_q4_k(w), kb.DTYPE_Q4_K
        ref = oracle.gemm_q4_k(blocks, x, M, N, K)
    assert rel_err(run(ctx, kb, torch_cuda, dt, blocks, x, N, kb.ACT_F32, shift), ref) <= 1e-3


@pytest.mark.parametrize("n", [1, 2047, 2048, 2049, 6147])
@pytest.mark.parametrize("shift", [0, 1])
def test_silu_mul(ctx, oracle, torch_cuda, n, shift):
    """Whole and partial groups of a CTA's 2048 elements, on 16 bytes and off them."""
    torch = torch_cuda
    g, u = (torch.randn(n + 4, generator=torch.Generator().manual_seed(n + i)) for i in (0, 1))
    gd, ud = g.cuda(), u.cuda()
    out = torch.full((n + 4,), float("nan"), device="cuda")
    ctx.silu_mul(gd[shift:], ud[shift:], out[shift:], n)
    ctx.sync()
    got = out.cpu().numpy()
    want = oracle.silu_mul(g[shift:shift + n].numpy(), u[shift:shift + n].numpy())
    assert rel_err(got[shift:shift + n], want) <= 1e-6
    assert (got[:shift] != got[:shift]).all() and (got[shift + n:] != got[shift + n:]).all()
