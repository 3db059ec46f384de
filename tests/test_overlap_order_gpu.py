"""GPU: with KANSO_OPT_OVERLAP_WEIGHT_PREFETCH on, calls read the caller's arrays only once the library
calls in front have written them. The option's promise is about the weight blocks of matmul calls alone.

A long addition keeps the stream busy; a short one behind it writes the array in question and lets its
dependents start at once, so that a read before the wait for it finds the old values.
"""
import ctypes

import numpy as np
import pytest

import plain_migurax as plain
import plain_revitar
from conftest import rel_err
from revitar_cases import to_bf16
from test_migurax_gpu import LatentCase, Memory, dev, f32, f64, guarded, unguard
from test_revitar_gpu import BF16, F32, PagedCase, to_dev, u32, unit_rows, up8

pytestmark = pytest.mark.gpu
BUSY = 1 << 28  # elements of the long addition: half a millisecond


@pytest.fixture(scope="module")
def eager(kb, torch_cuda):
    """A context with the option on, and a function that has an array written late."""
    torch = torch_cuda
    ctx = kb.Context(0, torch.cuda.current_stream())
    ctx.set_option(kb.OPT_OVERLAP_WEIGHT_PREFETCH, 1)
    big, one = torch.zeros(BUSY, device="cuda"), torch.ones(BUSY, device="cuda")

    def late(values):
        """A zeroed array of four-byte words (`values`' kind) that the stream will have filled."""
        words = dev(torch, values) if values.dtype == np.float32 else u32(torch, values)
        out = torch.zeros_like(words)
        torch.cuda.synchronize()
        ctx.call("kanso_cuda_residual_add", big.data_ptr(), one.data_ptr(), BUSY)
        # 0 + x is x, also where the words of small integers are read as (subnormal) floats
        ctx.call("kanso_cuda_residual_add", out.data_ptr(), words.data_ptr(), words.numel())
        return out, words

    yield ctx, late
    ctx.close()


@pytest.mark.parametrize("width", [64, 2048, 2052, 50])
@pytest.mark.parametrize("after", [0, 1])
def test_residual_norm(eager, torch_cuda, width, after):
    (ctx, late), torch = eager, torch_cuda
    rng = np.random.Generator(np.random.PCG64(width))
    x, y, w = (f32(rng.standard_normal(s)) for s in ((7, width), (7, width), width))
    xd, yd = guarded(torch, 7, width), dev(torch, y)
    xd[:7] = dev(torch, x)
    wd, keep = late(w)
    ctx.call("kanso_cuda_residual_norm", xd.data_ptr(), yd.data_ptr(), wd.data_ptr(), 1e-6, 1.7,
             after, 7, width)
    ref = (plain.rms_norm(1.7 * f64(x) + y, f64(w), 1e-6) if after else
           x + 1.7 * plain.rms_norm(f64(y), f64(w), 1e-6))
    assert rel_err(unguard(ctx, xd), ref) <= 1e-6


@pytest.mark.parametrize("H, G, D, DV", [(6, 2, 24, 16), (6, 2, 20, 12), (16, 4, 128, 128),
                                         (24, 8, 128, 128)])
@pytest.mark.parametrize("which", ["q", "k"])
def test_qk_norm_store(kb, eager, torch_cuda, H, G, D, DV, which):
    (ctx, late), torch = eager, torch_cuda
    rng = np.random.Generator(np.random.PCG64(H * D))
    T, bs, eps, ld, one = 5, 4, 0.3, up8(D), lambda v: np.array([v], np.uint32)
    qkv = f32(rng.standard_normal((T, H * D + G * D + G * DV)))
    qn, kn = f32(rng.standard_normal(H * D)), f32(rng.standard_normal(G * D))
    pool = kb.KvPool.dense(ctx, one(G), one(D), one(DV), 4, bs, kb.KV_F32)
    q_out = guarded(torch, T, H * ld)
    src = dev(torch, qkv)
    pos, seq, tab = u32(torch, np.arange(T)), u32(torch, np.zeros(T)), u32(torch, [2, 1, 0, 3])
    norms = [dev(torch, qn), dev(torch, kn)]
    at = "qk".index(which)
    norms[at], keep = late((qn, kn)[at])
    ctx.call("kanso_cuda_qk_norm_store", pool.h, 0, src.data_ptr(), norms[0].data_ptr(),
             norms[1].data_ptr(), eps, H, pos.data_ptr(), seq.data_ptr(), tab.data_ptr(), 4, T,
             q_out.data_ptr())
    ref = plain.rms_norm(f64(qkv[:, :H * D]), f64(qn), eps).reshape(T, H, D)
    assert rel_err(unguard(ctx, q_out).reshape(T, H, ld)[:, :, :D], ref) <= 1e-6
    if which == "k":
        # the stored keys, seen through the scores of queries that equal them (one visible key, no cap)
        q = np.zeros((1, H, ld), np.float32)
        k = plain.rms_norm(f64(qkv[:, H * D:H * D + G * D]), f64(kn), eps).reshape(T, G, D)[0]
        q[0, :, :D] = np.repeat(k, H // G, axis=0)
        out = guarded(torch, 1, H * DV)
        z = np.zeros(H, np.float32)
        p = kb.SigmoidAttentionParams(1, H, 4, 1, D ** -0.5, 0.0, z.ctypes.data, z.ctypes.data,
                                      z.ctypes.data)
        qd = dev(torch, q)
        ctx.call("kanso_cuda_sigmoid_attention", pool.h, 0, qd.data_ptr(), pos.data_ptr(),
                 seq.data_ptr(), tab.data_ptr(), out.data_ptr(), ctypes.byref(p), 1)
        score = np.repeat((k * k).sum(1), H // G) * D ** -0.5
        v = f64(qkv[0, H * D + G * D:]).reshape(G, DV)
        want = np.repeat(v, H // G, axis=0) / (1 + np.exp(-score))[:, None]
        assert rel_err(unguard(ctx, out).reshape(H, DV), want) <= 5e-6
    pool.destroy()


@pytest.mark.parametrize("V", [37, 64, 512, 516])
def test_head_norm_gate(eager, torch_cuda, V):
    (ctx, late), torch = eager, torch_cuda
    rng = np.random.Generator(np.random.PCG64(V))
    T, H, D, eps = 5, 4, 4, 0.2
    o, w = f32(rng.standard_normal((T, H, V))), f32(rng.standard_normal(H * V))
    y = f32(rng.standard_normal((T, H * (2 * D + 2 * V + 2))) * 3)
    out, od, yd = guarded(torch, T, H * V), dev(torch, o), dev(torch, y)
    wd, keep = late(w)
    ctx.call("kanso_cuda_head_norm_gate", od.data_ptr(), yd.data_ptr(), wd.data_ptr(), eps,
             out.data_ptr(), T, H, D, V)
    gate = y[:, H * (2 * D + V):H * (2 * D + 2 * V)]
    assert rel_err(unguard(ctx, out), plain.head_norm_gate(f64(o), f64(gate), f64(w), eps)) <= 2e-6


@pytest.mark.parametrize("compute", [F32, BF16])
@pytest.mark.parametrize("which", ["positions", "tables"])
def test_sigmoid_attention(kb, eager, torch_cuda, compute, which):
    (ctx, late), torch = eager, torch_cuda
    rng = np.random.Generator(np.random.PCG64(3))
    n, H, G, D, DV, T, window = 300, 6, 3, 64, 64, 5, 100
    k, v = unit_rows(rng.standard_normal((n, G, D))), to_bf16(rng.standard_normal((n, G, DV)))
    q, at = to_bf16(rng.standard_normal((T, H, D))), np.array([299, 40, 7, 160, 220])
    case = PagedCase(kb, ctx, torch, rng, k, v, 16, compute, H)
    z = np.zeros(H, np.float32)
    p = kb.SigmoidAttentionParams(T, H, case.nb, window, D ** -0.5, 5.0, z.ctypes.data, z.ctypes.data,
                                  z.ctypes.data)
    qd, out, seq = to_dev(torch, q, compute), guarded(torch, T, H * DV), u32(torch, np.zeros(T))
    pos, tab = u32(torch, at), case.tables
    if which == "positions":
        pos, keep = late(at.astype(np.uint32))
    else:
        tab, keep = late(case.table)
    ctx.call("kanso_cuda_sigmoid_attention", case.pool.h, 0, qd.data_ptr(), pos.data_ptr(),
             seq.data_ptr(), tab.data_ptr(), out.data_ptr(), ctypes.byref(p), 1)
    kk = f64(k if compute == F32 else to_bf16(k))
    ref = plain_revitar.attention_core(f64(q), kk, f64(v), at, np.arange(n), D ** -0.5, 5.0, f64(z),
                                       f64(z), f64(z), window)
    assert rel_err(unguard(ctx, out).reshape(T, H, DV), ref) <= (5e-6 if compute == F32 else 1e-2)
    case.pool.destroy()


@pytest.mark.parametrize("compute", [F32, BF16])
@pytest.mark.parametrize("which", ["positions", "tables"])
def test_latent_store_and_attention(kb, eager, torch_cuda, compute, which):
    (ctx, late), torch = eager, torch_cuda
    rng = np.random.Generator(np.random.PCG64(4))
    n, H, rank, rot, dim, T, bs, base = 300, 3, 64, 16, 7, 4, 16, 500.0
    raw, c_norm = rng.standard_normal((n, rank + rot)), f32(rng.uniform(0.5, 1.5, rank))
    case = LatentCase(kb, ctx, torch, rng, raw, c_norm, rank, base, bs, compute)
    tol = 1e-5 if compute == F32 else 2e-2

    def one_late(at):
        """Positions and tables, one of them written late."""
        pos, tab = u32(torch, at), case.tables
        if which == "positions":
            pos, keep = late(at.astype(np.uint32))
        else:
            tab, keep = late(case.tables.cpu().numpy().astype(np.uint32))
        return pos, tab, keep

    # the last rows once more, with other values
    at = np.arange(n - T, n)
    raw[at] = rng.standard_normal((T, rank + rot))
    down, qn = f32(np.concatenate([rng.standard_normal((T, 13)), raw[at]], 1)), np.ones(13, np.float32)
    arrays, seq = [dev(torch, a) for a in (down, qn, c_norm)], u32(torch, np.zeros(T))
    cq = torch.zeros(T * 32, device="cuda")
    p = case.params(T, 1, 1, 1.0, None)
    pos, tab, keep = one_late(at)
    ctx.call("kanso_cuda_latent_store", case.pool.h, 0, arrays[0].data_ptr(), 13,
             arrays[1].data_ptr(), arrays[2].data_ptr(), 1e-5, pos.data_ptr(), seq.data_ptr(),
             tab.data_ptr(), ctypes.byref(p), cq.data_ptr())
    case.c = plain.rms_norm(f64(f32(raw[:, :rank])), f64(c_norm), 1e-5)
    case.k_rot = plain.rotate(f64(f32(raw[:, rank:])), np.arange(n), base)

    at = np.array([299, 296, 20, 150])
    q_lat, q = rng.standard_normal((T, H, rank)) * 3, rng.standard_normal((T, H, dim + rot)) * 3
    sink, out = f32(rng.uniform(-1, 1, H)), guarded(torch, T, H * rank)
    ql, qq = dev(torch, q_lat), dev(torch, q)
    p = case.params(T, H, dim, 0.1, sink)
    pos, tab, keep = one_late(at)
    ctx.call("kanso_cuda_latent_attention", case.pool.h, 0, ql.data_ptr(), qq.data_ptr(),
             pos.data_ptr(), seq.data_ptr(), tab.data_ptr(), out.data_ptr(), ctypes.byref(p), 0)
    got = unguard(ctx, out).reshape(T, H, rank)
    assert rel_err(got, case.reference(q_lat, q, at, 0.1, sink)) <= tol
    case.pool.destroy()


@pytest.mark.parametrize("rows, hidden", [(3, 50), (3, 960), (3, 2048), (3, 5000), (700, 960)])
@pytest.mark.parametrize("which", ["x", "w"])
def test_rmsnorm(eager, torch_cuda, rows, hidden, which):
    (ctx, late), torch = eager, torch_cuda
    rng = np.random.Generator(np.random.PCG64(hidden))
    x, w = f32(rng.standard_normal((rows, hidden))), f32(rng.standard_normal(hidden))
    xd, wd, out = dev(torch, x), dev(torch, w), guarded(torch, rows, hidden)
    if which == "x":
        xd, keep = late(x)
    else:
        wd, keep = late(w)
    ctx.call("kanso_cuda_rmsnorm", xd.data_ptr(), wd.data_ptr(), out.data_ptr(), rows, hidden, 1e-5)
    assert rel_err(unguard(ctx, out), plain.rms_norm(f64(x), f64(w), 1e-5)) <= 2e-6


@pytest.mark.parametrize("n", [100, 5000])
@pytest.mark.parametrize("which", [0, 1])
def test_silu_mul(eager, torch_cuda, n, which):
    (ctx, late), torch = eager, torch_cuda
    rng = np.random.Generator(np.random.PCG64(n))
    a = [f32(rng.standard_normal(n)) for _ in range(2)]
    d, out = [dev(torch, v) for v in a], guarded(torch, 1, n)
    d[which], keep = late(a[which])
    ctx.call("kanso_cuda_silu_mul", d[0].data_ptr(), d[1].data_ptr(), out.data_ptr(), n)
    g = f64(a[0])
    assert rel_err(unguard(ctx, out)[0], g / (1 + np.exp(-g)) * a[1]) <= 1e-6


@pytest.mark.parametrize("compute, path, T, rows", [(F32, 1, 2, 50), (F32, 2, 40, 50), (BF16, 1, 2, 50),
                                                    (BF16, 2, 40, 300), (BF16, 2, 100, 14400)])
def test_bias_of_a_product(eager, torch_cuda, compute, path, T, rows):
    (ctx, late), torch = eager, torch_cuda
    rng = np.random.Generator(np.random.PCG64(rows))
    w, x, b = (f32(to_bf16(rng.standard_normal(s))) for s in ((rows, 72), (T, 72), rows))
    wd, xd, y = to_dev(torch, w, compute), to_dev(torch, x, compute), guarded(torch, T, rows)
    bd, keep = late(b)
    ctx.call("kanso_cuda_dense_linear_act", compute, wd.data_ptr(), xd.data_ptr(), bd.data_ptr(), 0,
             y.data_ptr(), T, rows, 72, path)
    assert rel_err(unguard(ctx, y), f64(x) @ f64(w).T + b) <= 4e-6


@pytest.mark.parametrize("which", ["router", "bias"])
@pytest.mark.parametrize("T, path", [(2, 1), (3, 2), (300, 2), (1300, 2)])
def test_router_of_experts(eager, torch_cuda, T, path, which):
    (ctx, late), torch = eager, torch_cuda
    rng = np.random.Generator(np.random.PCG64(T))
    experts, width, ff = 6, 64, 24
    w = {"router": to_bf16(np.eye(experts, width) * 6), "router.b": f32(np.arange(experts) * 0.01)}
    for e in range(experts):
        w[f"e{e}.up"] = to_bf16(rng.standard_normal((ff, width)) * width ** -0.5)
        w[f"e{e}.down"] = to_bf16(rng.standard_normal((width, ff)) * ff ** -0.5)
    x = to_bf16(rng.standard_normal((T, width)))
    x[:, :experts] = np.stack([rng.permutation(experts) for _ in range(T)])  # no close calls
    stack = lambda n: dev(torch, np.stack([w[f"e{e}.{n}"] for e in range(experts)]))
    xd, up, down, y = dev(torch, x), stack("up"), stack("down"), guarded(torch, T, width)
    router, bias = dev(torch, w["router"]), dev(torch, w["router.b"])
    if which == "router":
        router, keep = late(f32(w["router"]))
    else:
        bias, keep = late(w["router.b"])
    ctx.call("kanso_cuda_moe_relu2", F32, xd.data_ptr(), router.data_ptr(), bias.data_ptr(),
             up.data_ptr(), down.data_ptr(), y.data_ptr(), T, width, ff, experts, 2, path)
    ref = plain.moe(f64(x), plain.doubles(w), "", {"router": {"experts": experts, "top": 2}})
    assert rel_err(unguard(ctx, y), ref) <= 4e-6


@pytest.mark.parametrize("rows, path", [(1, 1), (20, 1), (130, 2)])
@pytest.mark.parametrize("which", ["y", "i", "f"])
def test_matrix_memory(kb, eager, torch_cuda, rows, path, which):
    """Projections and gate biases written late, from a state that a call before left."""
    (ctx, late), torch = eager, torch_cuda
    rng = np.random.Generator(np.random.PCG64(rows))
    H, D, V, before = 2, 24, 40, 30
    m = Memory(kb, ctx, torch, H, D, V, 9.0)
    a = m.inputs(rng, before + rows)
    ib, fb = f32(rng.standard_normal(H)), f32(rng.standard_normal(H))
    y = f32(np.concatenate([x.reshape(before + rows, -1) for x in a], axis=1))

    def call(part, pos0, path, is_late):
        n = part.shape[0]
        given = {"y": part, "i": ib, "f": fb}
        arrays = {k: dev(torch, v) for k, v in given.items()}
        out, p = guarded(torch, n, H * V), kb.MlstmParams(n, pos0, 0, m.cap)
        if is_late:
            arrays[which], keep = late(f32(given[which]))
        ctx.call("kanso_cuda_mlstm", m.pool.h, 0, arrays["y"].data_ptr(), arrays["i"].data_ptr(),
                 arrays["f"].data_ptr(), out.data_ptr(), ctypes.byref(p), path)
        return unguard(ctx, out).reshape(n, H, V)

    call(y[:before], 0, 1, False)
    got = call(y[before:], before, path, True)
    ref = m.reference(*a[:4], a[4] + ib, a[5] + fb)[before:]
    assert m.close(got, ref, 1e-4 if path == 1 else 5e-3)
    m.pool.destroy()
