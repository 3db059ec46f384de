"""GPU: products by pairs of CTAs (csrc/gemm_pair.cu) at the edges of their tiles (256 weight rows, 96 to
256 activation rows in multiples of 32, stages of 64 columns), against float64.

Tolerances as in test_revitar_gpu.py: bfloat16 products are exact in the f32 sum; the experts'
activations are rounded to bfloat16 once, 2^-8 of each value.
"""
import numpy as np
import pytest

import plain_revitar as plain
from conftest import rel_err
from revitar_cases import to_bf16
from test_revitar_gpu import BF16, padded, to_dev, up8

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T, rows, cols", [
    (96, 14400, 72),    # the fewest rows of a tile, one and a bit stages
    (97, 14340, 64),    # the same with one row over, weight rows past a multiple of 256
    (257, 7300, 1030),  # two tiles of rows, the second nearly as large
    (1000, 4099, 200),  # parts that leave a short last one
    (2048, 3072, 520),
])
def test_linear(ctx, torch_cuda, T, rows, cols):
    torch = torch_cuda
    rng = np.random.Generator(np.random.PCG64(T + rows))
    w, x = to_bf16(rng.standard_normal((rows, cols))), to_bf16(rng.standard_normal((T, cols)))
    bias = (rng.standard_normal(rows) * 5).astype(np.float32)
    wd, xd = (to_dev(torch, padded(a, up8(cols)), BF16) for a in (w, x))
    bd = torch.from_numpy(bias).cuda()
    ref = x.astype(np.float64) @ w.astype(np.float64).T
    for act in (False, True):
        y = torch.full((T + 1, rows), float("nan"), device="cuda")
        if act:
            ctx.call("kanso_cuda_dense_linear_act", BF16, wd.data_ptr(), xd.data_ptr(),
                     bd.data_ptr(), 1, y.data_ptr(), T, rows, cols, 2)
        else:
            ctx.call("kanso_cuda_dense_linear", BF16, wd.data_ptr(), xd.data_ptr(), y.data_ptr(), T,
                     rows, cols, 2)
        ctx.sync()
        got = y.cpu().numpy()
        want = np.maximum(ref + bias, 0) ** 2 if act else ref
        assert rel_err(got[:T], want) <= 4e-6 and np.isnan(got[T]).all()


@pytest.mark.parametrize("T, experts, top, lean", [(600, 3, 2, 0.0), (500, 4, 2, 3.0)])
def test_moe(ctx, torch_cuda, T, experts, top, lean):
    """Groups of any size, tiles that end inside them; `lean`: a favourite, others with few rows."""
    torch = torch_cuda
    rng = np.random.Generator(np.random.PCG64(T * 7 + experts))
    width, ff = 3080, 3200
    router = to_bf16(rng.standard_normal((experts, width)) * 3 * width ** -0.5)
    x = to_bf16(rng.standard_normal((8 * T, width)) + lean * router[:1])
    w = {"router": router}
    for e in range(experts):
        for n, s in (("gate", (ff, width)), ("up", (ff, width)), ("down", (width, ff))):
            w[f"e{e}.{n}"] = to_bf16(rng.standard_normal(s) * s[1] ** -0.5)
    s = np.sort(x.astype(np.float64) @ router.T.astype(np.float64), axis=1)[:, ::-1]
    x = x[np.argsort(s[:, top] - s[:, top - 1])[:T]]  # choices that are not a close call
    stack = lambda n: np.stack([w[f"e{e}.{n}"] for e in range(experts)])
    rd = torch.from_numpy(padded(router, up8(width))).cuda()
    gate, up, down = (to_dev(torch, padded(stack(n), up8(width if n != "down" else ff)), BF16)
                      for n in ("gate", "up", "down"))
    ref = plain.moe(x.astype(np.float64), {k: v.astype(np.float64) for k, v in w.items()}, "",
                    {"router": {"experts": experts, "top": top}})
    y = torch.full((T + 1, width), float("nan"), device="cuda")
    xd = torch.from_numpy(x).cuda()
    ctx.call("kanso_cuda_moe", BF16, xd.data_ptr(), rd.data_ptr(), gate.data_ptr(), up.data_ptr(),
             down.data_ptr(), y.data_ptr(), T, width, ff, experts, top, 2)
    ctx.sync()
    got = y.cpu().numpy()
    assert rel_err(got[:T], ref) <= 1e-2 and np.isnan(got[T]).all()
