"""GPU: products by pairs of CTAs (csrc/gemm_pair.cu) at the edges of their tiles (256 weight rows, 96 to
256 activation rows in multiples of 32, stages of 64 columns), against float64.

Tolerances as in test_revitar_gpu.py: bfloat16 products are exact in the f32 sum; the experts'
activations are rounded to bfloat16 once, 2^-8 of each value.

Which kernel takes a product depends on its sizes and on the number of SMs; by_pairs() says so here, so that a
case that no longer reaches the pairs fails instead of passing on the other kernel.
"""
import numpy as np
import pytest

import plain_migurax
import plain_revitar as plain
from conftest import rel_err
from migurax_cases import config, latent
from revitar_cases import to_bf16
from test_migurax_gpu import MiguraxCase
from test_revitar_gpu import BF16, padded, to_dev, up8

pytestmark = pytest.mark.gpu


def by_pairs(kb, ctx, rows, cols, T, groups=1, routed=False, gated=False):
    """launch_gemm_pair's choice (csrc/gemm_pair.cu): T rows in all, `routed`: shares on the device."""
    pairs, up = ctx.sm_count // 2, lambda a, b: -(-a // b)
    col_tiles, per = up(rows, 128 if gated else 256), T // groups
    if routed:
        return per >= 96 and 4 * col_tiles * up(T, 256) >= 3 * pairs
    cost = lambda parts, n: up(col_tiles * groups * parts, pairs) * (max((4096 + 16 * n) // 55, n // 2) + 16)
    sizes = [(p, up(up(per, p), 32) * 32) for p in range(up(per, 256), per // 96 + 1)]
    if not sizes:
        return False
    n = min(sizes, key=lambda s: cost(*s))[1]
    tiles = col_tiles * groups * up(per, n)
    if 4 * tiles < 3 * pairs:
        return False
    one_wave = up(rows, 128) * groups * up(per, 128) <= 2 * ctx.sm_count
    return not (one_wave and (tiles > pairs or (n == 256 and cols <= 1024)))


@pytest.mark.parametrize("T, rows, cols", [
    (96, 14400, 72),    # the fewest rows of a tile, one and a bit stages
    (97, 14340, 64),    # the same with one row over, weight rows past a multiple of 256
    (257, 7300, 1030),  # two tiles of rows, the second nearly as large
    (1000, 4099, 200),  # parts that leave a short last one
    (2048, 3072, 520),
    (1300, 4099, 200),  # as 1000, behind one wave
])
def test_linear(kb, ctx, torch_cuda, T, rows, cols):
    torch = torch_cuda
    assert by_pairs(kb, ctx, rows, cols, T) == ((T, rows) != (1000, 4099))  # that one in a single wave of CTAs
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


@pytest.mark.parametrize("T, experts, top, lean", [(600, 3, 2, 0.0), (500, 4, 2, 3.0), (620, 4, 2, 3.0)])
def test_moe(kb, ctx, torch_cuda, T, experts, top, lean):
    """Groups of any size, tiles that end inside them; `lean`: a favourite, others with few rows."""
    torch = torch_cuda
    assert by_pairs(kb, ctx, 3200, 3080, T * top, experts, True, True)
    assert by_pairs(kb, ctx, 3080, 3200, T * top, experts, True) == (T > 500)
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


def test_moe_of_many_experts(kb, ctx, torch_cuda):
    """More experts than a warp looks through at once, squared ReLU into rows with pads (ff is no multiple of
    eight), experts without rows and with one, at either end and in the middle."""
    torch = torch_cuda
    width, ff, experts = 1100, 1107, 41
    counts = np.full(experts, 115)
    counts[[0, 5, 31, 33, 40]] = 0
    counts[[1, 32, 39]] = 1
    counts[2] = 512
    T = int(counts.sum())
    assert T >= 96 * experts
    assert by_pairs(kb, ctx, ff, width, T, experts, True) and by_pairs(kb, ctx, width, ff, T, experts, True)
    rng = np.random.Generator(np.random.PCG64(41))
    want = rng.permutation(np.repeat(np.arange(experts), counts))  # the expert of each row, by construction
    router = np.zeros((experts, width))
    router[np.arange(experts), np.arange(experts)] = 4.0
    x = rng.standard_normal((T, width)) * 0.5
    x[:, :experts] = 0.0
    x[np.arange(T), want] = 3.0
    x, router = to_bf16(x), to_bf16(router)
    w = {"router": router, "router.b": np.zeros(experts, np.float32)}
    for e in range(experts):
        w[f"e{e}.up"] = to_bf16(rng.standard_normal((ff, width)) * width ** -0.5)
        w[f"e{e}.down"] = to_bf16(rng.standard_normal((width, ff)) * ff ** -0.5)
    stack = lambda n, ld: to_dev(torch, padded(np.stack([w[f"e{e}.{n}"] for e in range(experts)]),
                                               up8(ld)), BF16)
    rd, up, down = (torch.from_numpy(padded(router, up8(width))).cuda(), stack("up", width),
                    stack("down", ff))
    bias, xd = torch.zeros(experts, device="cuda"), torch.from_numpy(x).cuda()
    ref = plain_migurax.moe(x.astype(np.float64), plain_migurax.doubles(w), "",
                            {"router": {"experts": experts, "top": 1}})
    y = torch.full((T + 1, width), float("nan"), device="cuda")
    ctx.call("kanso_cuda_moe_relu2", BF16, xd.data_ptr(), rd.data_ptr(), bias.data_ptr(),
             up.data_ptr(), down.data_ptr(), y.data_ptr(), T, width, ff, experts, 1, 2)
    ctx.sync()
    got = y.cpu().numpy()
    assert rel_err(got[:T], ref) <= 1e-2 and np.isnan(got[T]).all()


class Heads(MiguraxCase):
    """One latent layer of 60 heads: products of one group for each head, without offsets."""
    models = {"heads": config(67, 64, [latent(60, 16, 8, 24, 30, 32, None)], alpha=1.2)}


@pytest.mark.parametrize("overlap", [1, 0])
def test_groups_of_heads_and_expanded_keys(kb, torch_cuda, tmp_path, overlap):
    """100 decoding sequences, alone and beside a long portion: key and value projections head by head (equal
    groups, results in bfloat16 side by side in a row, and by a list of rows), keys and values of a prompt
    expanded in one product (bfloat16 results)."""
    ctx = kb.Context(0, torch_cuda.cuda.current_stream())
    ctx.set_option(kb.OPT_OVERLAP_WEIGHT_PREFETCH, overlap)
    n, long = 100, 700
    for keys in (30, 24):  # rank columns of the key projection's results, value columns of the other's
        assert by_pairs(kb, ctx, keys, 64, 60 * n, 60)
    assert by_pairs(kb, ctx, 60 * (16 + 24), 30, long)
    c = Heads(kb, ctx, tmp_path, "heads", BF16, seed=7)
    e = kb.Engine(c.model, 4096, n + 1)
    reqs = [c.tokens(4) for _ in range(n)]
    refs = [c.plain(t) for t in reqs]
    prompt = c.tokens(long)
    whole = c.plain(prompt)
    logits = lambda r: np.frombuffer(r, np.float32).reshape(-1, c.V).copy()
    e.step([(i, t[:2], []) for i, t in enumerate(reqs)], c.V)
    # decoding alone
    got = logits(e.step([(i, t[2:3], [0]) for i, t in enumerate(reqs)], c.V))
    assert c.close(got, np.stack([r[2] for r in refs]), np.full(n, np.inf))
    # beside a prompt, in the middle of the decoding rows
    entries = [(i, t[3:4], [0]) for i, t in enumerate(reqs)]
    entries.insert(37, (n, prompt, list(range(long))))
    got = logits(e.step(entries, c.V))
    assert c.close(got[37:37 + long], whole)
    assert c.close(np.delete(got, np.s_[37:37 + long], 0), np.stack([r[3] for r in refs]),
                   np.full(n, np.inf))
    for i in range(n + 1):
        e.end(i)
    e.destroy()
    c.done()
    ctx.close()
