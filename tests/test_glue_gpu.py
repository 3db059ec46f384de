"""GPU: the row kernels of csrc/glue.cu at the borders of their forms: whole and partial groups of a CTA's
2048 elements; rows that a thread keeps one or four float4 of, wider ones and ragged ones; arrays on 16 bytes
and off them."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


def place(torch, values, off):
    """`values` behind `off` elements of NaN, and two behind them."""
    buf = torch.full((values.size + off + 2,), float("nan"), device="cuda")
    buf[off:off + values.size] = torch.from_numpy(values.reshape(-1)).cuda()
    return buf, buf[off:]


@pytest.mark.parametrize("n", [1, 2047, 2048, 2049, 6147])
@pytest.mark.parametrize("offs", [(0, 0), (1, 0), (0, 3), (2, 2)])
def test_residual_add(ctx, torch_cuda, n, offs):
    rng = np.random.Generator(np.random.PCG64(n))
    h, p = (rng.standard_normal(n).astype(np.float32) for _ in range(2))
    (hb, hd), (_, pd) = (place(torch_cuda, a, o) for a, o in zip((h, p), offs))
    ctx.residual_add(hd, pd, n)
    ctx.sync()
    got = hb.cpu().numpy()
    assert (got[offs[0]:offs[0] + n] == h + p).all()  # one rounding: exact
    assert np.isnan(got[:offs[0]]).all() and np.isnan(got[offs[0] + n:]).all()


@pytest.mark.parametrize("rows, hidden", [(5, h) for h in (1, 50, 64, 1000, 1024, 1028, 4096, 4100, 8192, 9001)] +
                         [(700, 4), (700, 1024)])  # more rows than four to an SM
@pytest.mark.parametrize("off", [None, "x", "w", "out"])
def test_rmsnorm(ctx, oracle, torch_cuda, rows, hidden, off):
    rng = np.random.Generator(np.random.PCG64(hidden))
    x, w = rng.standard_normal((rows, hidden)).astype(np.float32), rng.standard_normal(hidden).astype(np.float32)
    (_, xd), (_, wd), (ob, od) = (place(torch_cuda, a, int(off == n)) for a, n in
                                  ((x, "x"), (w, "w"), (np.zeros_like(x), "out")))
    ctx.rmsnorm(xd, wd, od, rows, hidden, 1e-5)
    ctx.sync()
    got = od.cpu().numpy()
    assert rel_err(got[:rows * hidden].reshape(rows, -1), oracle.rmsnorm(x, w, 1e-5)) <= 2e-6
    assert np.isnan(got[rows * hidden:]).all() and int(torch_cuda.isnan(ob).sum()) == 2 + int(off == "out")
