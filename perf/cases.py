"""The work that a user of this library has it do, as timed cases over its public entry points.

Five kinds, each with the sizes it stands for:
  ffn      a gated feed-forward block on quantised weights (gate, up, silu * up, down), which is how
           LinearWeight::forward is called outside of the decode step; 1 to 512 rows.
  chunk    a portion of a prompt over the quantised pool: its K and V rows are stored, then attended.
  llama    one decode step of a quantised llama model, one token per sequence.
  prompt   a ragged step of an unquantised model: portions of prompts, beside decoding sequences.
  decode   one decode step of an unquantised model.

Values come from the seed alone; row counts, context lengths and layers come from the case.
"""
import importlib
import json
import math
import os
import tempfile

import numpy as np
import torch

kb = importlib.import_module("kanso-infer_b200").backend

BS = 16  # tokens per page, everywhere

# width, query heads, key/value heads, feed-forward width, vocabulary of the llama models
LLAMA = {"360m": (960, 15, 5, 2560, 49152), "1k": (1024, 16, 4, 2048, 32768),
         "2k": (2048, 16, 4, 4096, 32768)}
VOCAB = 32768
# width, query heads, key/value heads, head size, window, experts, chosen, expert width
REVITAR = {"1k": (1024, 16, 4, 64, 1024, 16, 2, 1024), "2k": (2048, 16, 4, 128, 2048, 16, 4, 1024)}
# heads, plain / rotated / value columns, both ranks; heads, key and value columns of the memory
MIGURAX = {"1k": (16, 64, 32, 64, 256, 384, 4, 128, 256),
           "2k": (16, 128, 64, 128, 512, 768, 4, 256, 512)}


def listed():
    return [
        # one token through the feed-forward of SmolLM2-360M: all latency
        dict(name="ffn_q8_0_960_m1", kind="ffn", fmt="q8_0", act="f32", width=960, ff=2560, rows=1),
        # one token through an 8B-class model's feed-forward: the weights' bytes
        dict(name="ffn_q4_k_4096_m1", kind="ffn", fmt="q4_k", act="f32", width=4096, ff=14336,
             rows=1),
        # a decoding batch through the same
        dict(name="ffn_q4_k_4096_m24", kind="ffn", fmt="q4_k", act="f32", width=4096, ff=14336,
             rows=24),
        # a portion of a prompt: tensor-core work
        dict(name="ffn_q8_0_4096_m512", kind="ffn", fmt="q8_0", act="f32", width=4096, ff=14336,
             rows=512),
        # activations quantised like the weights, exact block sums
        dict(name="ffn_q8_0_q8_m100", kind="ffn", fmt="q8_0", act="q8", width=4096, ff=14336,
             rows=100),
        # chunked prefill of four requests over the int8 pool, SmolLM2-360M's heads
        dict(name="chunk_int8_4x512", kind="chunk", pool="int8", heads=15, kv_heads=5, dim=64,
             seqs=4, rows=2048, cached=1536),
        # decoding with SmolLM2-360M: alone, and a full batch with uneven contexts
        dict(name="llama_360m_b1", kind="llama", model="360m", fmt="q8_0", layers=32, pool="int8",
             seqs=1, ctx_min=1673, ctx_max=1673),
        dict(name="llama_360m_b64", kind="llama", model="360m", fmt="q8_0", layers=32, pool="int8",
             seqs=64, ctx_min=256, ctx_max=4096),
        # unquantised models: a long prompt's second half, a mixed step, decoding batches
        dict(name="revitar_2k_prompt", kind="prompt", arch="Revitar", size="2k", layers=4, seqs=1,
             rows=2048, cached=2048, decoding=0),
        dict(name="migurax_2k_mixed", kind="prompt", arch="Migurax", size="2k", layers=4, seqs=3,
             rows=2040, cached=512, decoding=8),
        dict(name="revitar_2k_decode_b8", kind="decode", arch="Revitar", size="2k", layers=4,
             seqs=8, ctx_min=700, ctx_max=4000),
        dict(name="migurax_2k_decode_b2", kind="decode", arch="Migurax", size="2k", layers=4,
             seqs=2, ctx_min=1000, ctx_max=2048),
    ]


def _log(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["ffn", "ffn", "ffn", "chunk", "llama", "llama", "prompt", "decode"])
    if kind == "ffn":
        fmt = rng.choice(["q8_0", "q4_k"])
        act = rng.choice(["f32", "f32", "q8"]) if fmt == "q8_0" else "f32"
        step = 32 if fmt == "q8_0" else 256
        if rng.random() < 0.6:
            width, ff = rng.choice([(960, 2560), (1024, 2048), (2048, 4096), (4096, 14336)]
                                   if fmt == "q8_0" else
                                   [(1024, 2048), (2048, 4096), (4096, 14336)])
        else:
            width = _log(rng, 512 // step, 4096 // step) * step
            ff = _log(rng, 1024 // step, 14336 // step) * step
        return dict(kind="ffn", fmt=fmt, act=act, width=width, ff=ff, rows=_log(rng, 1, 512))
    if kind == "chunk":
        heads, kv, dim = rng.choice([(15, 5, 64), (16, 4, 64), (16, 4, 128), (32, 8, 128)])
        seqs = rng.randint(1, 6)
        return dict(kind="chunk", pool=rng.choice(["int8", "int8", "fp8"]), heads=heads,
                    kv_heads=kv, dim=dim, seqs=seqs, rows=_log(rng, 8 * seqs, 1500),
                    cached=rng.choice([0, _log(rng, 16, 1536)]))
    if kind == "llama":
        model = rng.choice(["360m", "360m", "1k", "2k"])
        top = _log(rng, 256, 4096)
        return dict(kind="llama", model=model,
                    fmt="q8_0" if model == "360m" else rng.choice(["q8_0", "q4_k"]),
                    layers=rng.randint(4, 32 if model == "360m" else 10),
                    pool=rng.choice(["int8", "int8", "fp8"]), seqs=_log(rng, 1, 64),
                    ctx_min=rng.randint(40, top), ctx_max=top)
    arch, size = rng.choice(["Revitar", "Migurax"]), rng.choice(["1k", "2k"])
    layers = rng.randint(2, 4)
    if kind == "prompt":
        seqs = rng.randint(1, 4)
        return dict(kind="prompt", arch=arch, size=size, layers=layers, seqs=seqs,
                    rows=_log(rng, 40 * seqs, 2040), cached=rng.choice([0, _log(rng, 16, 1536)]),
                    decoding=rng.choice([0, rng.randint(1, 24)]))
    seqs = _log(rng, 1, 48)
    top = _log(rng, 128, min(4096, 24576 // seqs))
    return dict(kind="decode", arch=arch, size=size, layers=layers, seqs=seqs,
                ctx_min=rng.randint(64, top), ctx_max=top)


# ---- what the cases are made of ----

_context = None


def _ctx():
    """One context per process, as a serving program keeps it; weights are uploaded once and left
    alone, which is what the option promises."""
    global _context
    if _context is None:
        torch.cuda.set_device(0)
        stream = torch.cuda.Stream()
        ctx = kb.Context(0, stream)
        ctx.set_option(kb.OPT_OVERLAP_WEIGHT_PREFETCH, 1)
        _context = (ctx, stream)
    return _context[0]


def _gen(seed, *path):
    g = torch.Generator(device="cuda")
    for p in path:
        seed = (seed * 1000003 + p + 12345) % (1 << 61)
    return g.manual_seed(seed)


def _normal(g, *shape):
    return torch.randn(shape, generator=g, device="cuda")


def _half_away(x):
    return torch.sign(x) * torch.floor(x.abs() + 0.5)


def _blocks(w, fmt):
    """GGUF blocks of a float matrix, uint8 [rows, bytes of a row]."""
    n, k = w.shape
    if fmt == "q8_0":
        v = w.view(n, k // 32, 32)
        d = (v.abs().amax(-1, keepdim=True) / 127).half()
        q = torch.clamp(_half_away(v / d.float().clamp_min(1e-30)), -127, 127).to(torch.int8)
        return torch.cat([d.view(torch.uint8), q.view(torch.uint8)], -1).view(n, -1)
    v = w.view(n, k // 256, 8, 32)
    low = (-v.amin(-1)).clamp_min(0)
    span = (v.amax(-1) + low) / 15
    d, m = (t.amax(-1, keepdim=True).div(63).half() for t in (span, low))
    sc, mn = (torch.clamp(torch.round(t / s.float().clamp_min(1e-30)), 0, 63).to(torch.uint8)
              for t, s in ((span, d), (low, m)))
    scale = (d.float() * sc).unsqueeze(-1)
    base = (m.float() * mn).unsqueeze(-1)
    q = torch.where(scale > 0, (v + base) / scale, torch.zeros_like(v))
    q = torch.clamp(torch.round(q), 0, 15).to(torch.uint8)
    head = torch.cat([sc[..., :4] | (sc[..., 4:] >> 4 << 6), mn[..., :4] | (mn[..., 4:] >> 4 << 6),
                      (sc[..., 4:] & 15) | (mn[..., 4:] & 15) << 4], -1)
    nib = q[..., 0::2, :] | q[..., 1::2, :] << 4
    return torch.cat([d.view(torch.uint8), m.view(torch.uint8), head, nib.flatten(-2)],
                     -1).view(n, -1)


def _values(blocks, fmt):
    """The numbers that blocks stand for, float64."""
    n = blocks.shape[0]
    if fmt == "q8_0":
        b = blocks.view(n, -1, 34)
        d = b[..., :2].contiguous().view(torch.float16).double()
        return (b[..., 2:].contiguous().view(torch.int8).double() * d).view(n, -1)
    b = blocks.view(n, -1, 144)
    d, m = (b[..., i:i + 2].contiguous().view(torch.float16).double() for i in (0, 2))
    lo, mid, hi = b[..., 4:8], b[..., 8:12], b[..., 12:16]
    sc = torch.cat([lo & 63, (hi & 15) | (lo >> 6) << 4], -1).double()
    mn = torch.cat([mid & 63, (hi >> 4) | (mid >> 6) << 4], -1).double()
    nib = b[..., 16:].reshape(n, -1, 4, 1, 32)
    q = torch.cat([nib & 15, nib >> 4], 3).view(n, -1, 8, 32).double()
    return ((d * sc).unsqueeze(-1) * q - (m * mn).unsqueeze(-1)).view(n, -1)


def _stored(x, pool):
    """float32 rows [..., dim] as a quantised pool keeps them, float64."""
    top = x.abs().amax(-1, keepdim=True)
    if pool == "int8":
        s = torch.where(top > 0, top / 127, torch.ones_like(top))
        return torch.clamp(_half_away(x * (1 / s)), -127, 127).double() * s.double()
    s = torch.where(top > 0, torch.exp2(torch.ceil(torch.log2(top / 64))), torch.ones_like(top))
    return (x / s).to(torch.float8_e4m3fn).double() * s.double()


def _lens(c):
    """The sequences' context lengths: spread evenly from ctx_min to ctx_max."""
    n, lo, hi = c["seqs"], c["ctx_min"], c["ctx_max"]
    return [hi - (hi - lo) * i // max(1, n - 1) for i in range(n)]


def _portions(c):
    """(context, query) lengths of a case's portions: uneven, `rows` in all."""
    n, rows = c["seqs"], c["rows"]
    cut = [rows * i * (i + n) // (n * (n + n)) for i in range(n + 1)]
    return [(c["cached"] * (i + 1) // n + b - a, b - a)
            for i, (a, b) in enumerate(zip(cut, cut[1:]))]


def _tables(lens, seed):
    """Block tables with the pages anywhere in the pool, padded with each sequence's last page."""
    n = [(x + BS - 1) // BS for x in lens]
    perm = np.random.Generator(np.random.PCG64(seed)).permutation(sum(n) + 4)
    tab, at = np.zeros((len(n), max(n)), np.uint32), 0
    for i, b in enumerate(n):
        tab[i, :b] = perm[at:at + b]
        tab[i, b:] = tab[i, b - 1]
        at += b
    return tab, len(perm)


def _slots(tab, i, first, end):
    t = np.arange(first, end)
    return tab[i][t // BS] * BS + t % BS


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a).astype(np.int32)).cuda()


def _u32(a):
    return np.ascontiguousarray(a, np.uint32)


# ---- ffn ----

def _ffn_data(c, seed):
    g, w, f = _gen(seed, 1), c["width"], c["ff"]
    mats = [_blocks(_normal(g, r, k) * 0.02, c["fmt"]) for r, k in ((f, w), (f, w), (w, f))]
    return mats, _normal(g, c["rows"], w)


def _ffn_prepare(c, seed):
    ctx, (mats, x) = _ctx(), _ffn_data(c, seed)
    w, f, m = c["width"], c["ff"], c["rows"]
    dt = kb.DTYPE_Q8_0 if c["fmt"] == "q8_0" else kb.DTYPE_Q4_K
    ws = [kb.Weight(ctx, b.cpu().numpy(), dt, r, k) for b, (r, k) in
          zip(mats, ((f, w), (f, w), (w, f)))]
    buf = [torch.empty(m, k, device="cuda") for k in (f, f, f, w)]
    return dict(ctx=ctx, ws=ws, x=x, buf=buf, m=m, n=m * f,
                act=kb.ACT_Q8 if c["act"] == "q8" else kb.ACT_F32)


def _ffn_run(s):
    (gate, up, down), (a, b, h, y), m = s["ws"], s["buf"], s["m"]
    gate.forward(s["x"], a, m, s["act"])
    up.forward(s["x"], b, m, s["act"])
    s["ctx"].silu_mul(a, b, h, s["n"])
    down.forward(h, y, m, s["act"])
    return a, b, y


def _q8(x):
    """Activations as quantize_row_q8_0 makes them, in its own 32-bit steps."""
    v = x.float().view(x.shape[0], -1, 32)
    d = v.abs().amax(-1, keepdim=True) / 127
    q = torch.clamp(_half_away(v * torch.where(d > 0, 1 / d, torch.zeros_like(d))), -128, 127)
    return (q.double() * d.double()).view(x.shape[0], -1)


def _ffn_exact(c, seed):
    mats, x = _ffn_data(c, seed)
    act = _q8 if c["act"] == "q8" else (lambda v: v)
    gate, up, down = (_values(b, c["fmt"]) for b in mats)
    x = act(x.double())
    a, b = x @ gate.T, x @ up.T
    return a, b, act(torch.nn.functional.silu(a) * b) @ down.T


def _ffn_work(c):
    n = 3 * c["width"] * c["ff"]
    byts = n // 32 * 34 if c["fmt"] == "q8_0" else n // 256 * 144
    return dict(bytes=byts + 4 * c["rows"] * (2 * c["width"] + 2 * c["ff"]),
                flops=2 * c["rows"] * n)


# ---- chunk ----

def _chunk_data(c, seed):
    lens, (tab, pages) = _portions(c), _tables([x for x, _ in _portions(c)], seed)
    g, kd = _gen(seed, 2), c["kv_heads"] * c["dim"]
    kv = [(_normal(g, n, kd), _normal(g, n, kd)) for n, _ in lens]
    return lens, tab, pages, kv, _normal(g, c["rows"], c["heads"] * c["dim"])


def _pool_type(c):
    return kb.KV_FP8 if c["pool"] == "fp8" else kb.KV_INT8


def _chunk_prepare(c, seed):
    ctx, (lens, tab, pages, kv, q) = _ctx(), _chunk_data(c, seed)
    pool = kb.KvPool(ctx, 1, pages, BS, c["kv_heads"], c["dim"], _pool_type(c))
    new = []
    torch.cuda.synchronize()
    for i, ((n, t), (k, v)) in enumerate(zip(lens, kv)):
        if n > t:
            pool.write_slots(0, _dev(_slots(tab, i, 0, n - t)), k[:n - t], v[:n - t], n - t)
            ctx.sync()
        new.append(_slots(tab, i, n - t, n))
    new = _u32(np.concatenate(new))
    k, v = (torch.cat([p[j][n - t:] for (n, t), p in zip(lens, kv)]).contiguous() for j in (0, 1))
    params = kb.PagedAttentionParams(len(lens), c["heads"], c["kv_heads"], c["dim"], BS,
                                     tab.shape[1], c["dim"] ** -0.5)
    return dict(pool=pool, new=_dev(new), new_host=new, k=k, v=v, q=q, rows=c["rows"],
                tab=_dev(tab), out=torch.empty_like(q), params=params,
                ctx_lens=_u32([n for n, _ in lens]), q_lens=_u32([t for _, t in lens]))


def _chunk_run(s):
    s["pool"].write_slots(0, s["new"], s["k"], s["v"], s["rows"], s["new_host"])
    s["pool"].paged_attention_prefill(0, s["q"], s["tab"], s["ctx_lens"], s["q_lens"], s["out"],
                                      s["params"])
    return s["out"]


def _causal(q, k, v, scale):
    """The last rows q [T, H, d] of a sequence with keys k [S, G, d]: float64 softmax attention."""
    T, S, rep = q.shape[0], k.shape[0], q.shape[1] // k.shape[1]
    seen = torch.arange(S, device="cuda") <= torch.arange(S - T, S, device="cuda")[:, None]
    out = []
    for g in range(k.shape[1]):
        p = torch.einsum("thd,sd->hts", q[:, g * rep:(g + 1) * rep], k[:, g]) * scale
        p = torch.softmax(p.masked_fill(~seen, -math.inf), -1)
        out.append(torch.einsum("hts,sd->thd", p, v[:, g]))
    return torch.cat(out, 1).reshape(T, -1)


def _chunk_exact(c, seed):
    lens, _, _, kv, q = _chunk_data(c, seed)
    out, at = [], 0
    for (n, t), (k, v) in zip(lens, kv):
        k, v = (_stored(x.view(n, c["kv_heads"], c["dim"]), c["pool"]) for x in (k, v))
        out.append(_causal(q[at:at + t].view(t, c["heads"], c["dim"]).double(), k, v,
                           c["dim"] ** -0.5))
        at += t
    return torch.cat(out)


def _chunk_work(c):
    H, G, d = c["heads"], c["kv_heads"], c["dim"]
    byts, flops = 8 * c["rows"] * H * d + 8 * c["rows"] * G * d, 0
    for n, t in _portions(c):
        byts += n * G * (2 * d + 8)
        flops += 4 * H * d * sum(range(n - t + 1, n + 1))
    return dict(bytes=byts, flops=flops)


# ---- llama ----

def _llama_shapes(c):
    W, H, G, F, V = LLAMA[c["model"]]
    d = W // H
    return [(H * d, W), (G * d, W), (G * d, W), (W, H * d), (F, W), (F, W), (W, F)]


def _llama_layer(c, seed, l):
    g, W = _gen(seed, 3, l), LLAMA[c["model"]][0]
    return ([_blocks(_normal(g, *s) * 0.02, c["fmt"]) for s in _llama_shapes(c)],
            [1 + 0.1 * _normal(g, W) for _ in range(2)])


def _llama_ends(c, seed):
    W, _, _, _, V = LLAMA[c["model"]]
    g = _gen(seed, 4)
    toks = np.random.Generator(np.random.PCG64(seed + 1)).integers(0, V, c["seqs"])
    return _blocks(_normal(g, V, W) * 0.02, "q8_0"), 1 + 0.1 * _normal(g, W), toks


def _llama_rows(c, seed, l, n):
    g, (W, H, G, _, _) = _gen(seed, 5, l), LLAMA[c["model"]]
    return [_normal(g, n, G * (W // H)) for _ in range(2)]


def _llama_prepare(c, seed):
    ctx, (W, H, G, F, V) = _ctx(), LLAMA[c["model"]]
    L, lens, dt = c["layers"], _lens(c), kb.DTYPE_Q8_0 if c["fmt"] == "q8_0" else kb.DTYPE_Q4_K
    m = kb.Model(ctx, kb.ModelConfig(W, H, G, L, F, V, BS, 4352, 1e-5, 100000.0))
    tab, pages = _tables(lens, seed)
    pool = kb.KvPool(ctx, L, pages, BS, G, W // H, _pool_type(c))
    hist = _dev(np.concatenate([_slots(tab, i, 0, n - 1) for i, n in enumerate(lens)]))
    for l in range(L):
        mats, norms = _llama_layer(c, seed, l)
        for which, (b, (r, k)) in enumerate(zip(mats, _llama_shapes(c))):
            m.set_weight(l, which, b.cpu().numpy(), dt, r, k)
        for which, w in enumerate(norms):
            m.set_norm(l, which, w.cpu().numpy())
        k, v = _llama_rows(c, seed, l, len(hist))
        torch.cuda.synchronize()
        pool.write_slots(l, hist, k, v, len(hist))
        ctx.sync()
    emb, norm, toks = _llama_ends(c, seed)
    m.set_weight(0, kb.W_TOKEN_EMBD, emb.cpu().numpy(), kb.DTYPE_Q8_0, V, W)
    m.set_norm(0, kb.NORM_FINAL, norm.cpu().numpy())
    pos = np.array(lens) - 1
    args = [_dev(a) for a in (toks, pos, [_slots(tab, i, p, p + 1)[0] for i, p in enumerate(pos)],
                              tab, lens)]
    return dict(m=m, pool=pool, args=args, B=len(lens), blocks=tab.shape[1], top=max(lens),
                logits=torch.empty(len(lens), V, device="cuda"))


def _step_run(s):
    s["m"].decode_step_device(s["pool"], *s["args"], s["B"], s["blocks"], s["top"], s["logits"])
    return s["logits"]


def _rms(x, w, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w.double()


def _llama_exact(c, seed):
    W, H, G, F, V = LLAMA[c["model"]]
    d, lens, silu = W // H, _lens(c), torch.nn.functional.silu
    emb, norm, toks = _llama_ends(c, seed)
    x = _values(emb[torch.from_numpy(toks).cuda()], "q8_0")
    freq = 100000.0 ** (-torch.arange(0, d, 2, device="cuda").double() / d)
    angle = (torch.tensor(lens, device="cuda").double() - 1)[:, None, None] * freq

    def rope(t):
        t = t.view(len(lens), -1, d)
        a, b = t[..., :d // 2], t[..., d // 2:]
        return torch.cat([a * angle.cos() - b * angle.sin(), b * angle.cos() + a * angle.sin()], -1)

    for l in range(c["layers"]):
        mats, norms = _llama_layer(c, seed, l)
        wq, wk, wv, wo, wg, wu, wd = (_values(b, c["fmt"]) for b in mats)
        h = _rms(x, norms[0], 1e-5)
        q, k, v = rope(h @ wq.T), rope(h @ wk.T), (h @ wv.T).view(len(lens), G, d)
        k, v = (_stored(t.float(), c["pool"]) for t in (k, v))
        kh, vh = _llama_rows(c, seed, l, sum(lens) - len(lens))
        out, at = [], 0
        for i, n in enumerate(lens):
            ki, vi = (torch.cat([_stored(t[at:at + n - 1].view(n - 1, G, d), c["pool"]), e[i:i + 1]])
                      for t, e in ((kh, k), (vh, v)))
            p = torch.softmax(torch.einsum("grd,sgd->grs", q[i].view(G, H // G, d), ki) * d ** -0.5,
                              -1)
            out.append(torch.einsum("grs,sgd->grd", p, vi).reshape(-1))
            at += n - 1
        x = x + torch.stack(out) @ wo.T
        h = _rms(x, norms[1], 1e-5)
        x = x + (silu(h @ wg.T) * (h @ wu.T)) @ wd.T
    return _rms(x, norm, 1e-5) @ _values(emb, "q8_0").T


def _llama_work(c):
    W, H, G, F, V = LLAMA[c["model"]]
    n = c["layers"] * sum(r * k for r, k in _llama_shapes(c))
    total, B = sum(_lens(c)), c["seqs"]
    byts = (n // 32 * 34 if c["fmt"] == "q8_0" else n // 256 * 144) + V * W // 32 * 34
    return dict(bytes=byts + c["layers"] * total * G * (2 * W // H + 8) + 4 * B * V,
                flops=2 * B * (n + V * W) + 4 * c["layers"] * total * W)


# ---- prompt, decode: the unquantised models ----

def _class_config(c):
    """config.json, and name -> (shape, how its values are made)."""
    W, H, G, D, win, E, top, F = REVITAR[c["size"]]
    shapes = {"embed": (VOCAB, W), "head": (VOCAB, W), "final.norm": (W,)}
    moe = {"kind": "moe", "expert": {"ff": F}, "router": {"experts": E, "top": top}}
    layers = []
    for i in range(c["layers"]):
        p, x, q = f"l{i}.", f"l{i}.mix.", f"l{i}.mlp."
        shapes.update({p + "norm1": (W,), p + "norm2": (W,)})
        if c["arch"] == "Revitar":
            layers.append({"type": "attention", "mlp": moe,
                           "mixer": {"heads": H, "kv_heads": G, "dim": D, "vdim": D,
                                     "scale": D ** -0.5, "softcap": 30.0, "mask": {"size": win}}})
            shapes.update({x + "q": (H * D, W), x + "k": (G * D, W), x + "v": (G * D, W),
                           x + "o": (W, H * D), x + "q.norm": (H * D,), x + "k.norm": (G * D,),
                           x + "r1": (H,), x + "r2": (H,), x + "pb": (H,)})
        else:
            h, d, rd, dv, r, qr, mh, md, mv = MIGURAX[c["size"]]
            mixer = ({"heads": h, "dim": d, "rot_dim": rd, "vdim": dv, "kv_rank": r, "q_rank": qr,
                      "scale": (d + rd) ** -0.5, "rot": {"base": 10000.0, "dims": rd}},
                     {"heads": mh, "dim": md, "vdim": mv, "gate_cap": 15.0})[i % 2]
            layers.append({"type": ("latent_attention", "mlstm")[i % 2], "mixer": mixer,
                           "mlp": moe if i else {"kind": "dense", "ff": top * F}})
            if i % 2 == 0:
                shapes.update({x + "dq": (qr, W), x + "dq.norm": (qr,), x + "uq": (h * (d + rd), qr),
                               x + "dkv": (r + rd, W), x + "dkv.norm": (r,), x + "uk": (h * d, r),
                               x + "uv": (h * dv, r), x + "sink": (h,), x + "o": (W, h * dv)})
            else:
                shapes.update({x + "k": (mh * md, W), x + "q": (mh * md, W), x + "v": (mh * mv, W),
                               x + "g": (mh * mv, W), x + "i": (mh, W), x + "f": (mh, W),
                               x + "i.b": (mh,), x + "f.b": (mh,), x + "norm": (mh * mv,),
                               x + "o": (W, mh * mv)})
            if i == 0:
                shapes.update({q + "up": (top * F, W), q + "up.b": (top * F,),
                               q + "down": (W, top * F), q + "down.b": (W,)})
                continue
            shapes[q + "router.b"] = (E,)
        shapes[q + "router"] = (E, W)
        for e in range(E):
            if c["arch"] == "Revitar":
                shapes[f"{q}e{e}.gate"] = (F, W)
            shapes[f"{q}e{e}.up"], shapes[f"{q}e{e}.down"] = (F, W), (W, F)
    cfg = {"architecture": c["arch"], "vocab": VOCAB, "width": W, "norm": {"eps": 1e-6},
           "layers": layers}
    cfg.update({"embedding": {"scale": 1.0}, "residual_mult": 0.7} if c["arch"] == "Revitar" else
               {"postln_alpha": 1.5})
    return cfg, shapes


def _class_weights(c, seed):
    """(config, name -> bfloat16 tensor). As in trained models a token's memory query leans towards its
    own key, the forget gates keep tens to hundreds of tokens, and a router has a clear favourite."""
    cfg, shapes = _class_config(c)
    g, w = _gen(seed, 6), {}
    for name, sh in shapes.items():
        t = _normal(g, *sh)
        if "norm" in name.split(".")[-1]:
            t = 1 + 0.1 * t
        elif name.endswith((".r1", ".r2")):
            t = 0.2 + 0.1 * t.abs()
        elif name.endswith((".pb", ".f.b")):
            t = t + (4 if name.endswith(".f.b") else -4)
        elif len(sh) > 1 and name != "embed":
            t = t * sh[-1] ** -0.5 * (4 if name.endswith("router") else 1)
            if c["arch"] == "Migurax" and name.endswith("mix.q"):
                t = 0.8 * t + 0.6 * w[name[:-1] + "k"].float()
        w[name] = t.to(torch.bfloat16)
    return cfg, w


def _class_model(ctx, c, seed):
    cfg, w = _class_weights(c, seed)
    header, at = {}, 0
    for name, t in w.items():
        header[name] = {"dtype": "BF16", "shape": list(t.shape),
                        "data_offsets": [at, at + 2 * t.numel()]}
        at += 2 * t.numel()
    text = json.dumps(header).encode()
    text += b" " * (-len(text) % 8)
    data = torch.cat([t.flatten() for t in w.values()]).view(torch.int16).cpu().numpy()
    fast = "/dev/shm"
    room = os.path.isdir(fast) and os.statvfs(fast).f_bavail * os.statvfs(fast).f_frsize > 2 * at
    with tempfile.TemporaryDirectory(dir=fast if room else None) as folder:
        with open(os.path.join(folder, "config.json"), "w") as f:
            json.dump(cfg, f)
        with open(os.path.join(folder, "model.safetensors"), "wb") as f:
            f.write(len(text).to_bytes(8, "little") + text)
            f.write(data)
        return kb.Model.from_dir(ctx, folder)


def _class_lens(c):
    """(context, query) lengths of all sequences of the step."""
    if c["kind"] == "decode":
        return [(n, 1) for n in _lens(c)]
    return _portions(c) + [(c["cached"] // 2 + 37 * (i + 1), 1) for i in range(c["decoding"])]


def _want(c):
    """Rows of a prompt step whose logits are asked for: each sequence's last one, and 24 of the
    portions' rows as a scoring program reads them."""
    last = np.cumsum([t for _, t in _class_lens(c)]) - 1
    return _u32(sorted({int(r) for r in last} | {c["rows"] * i // 24 for i in range(24)}))


def _class_tokens(c, seed):
    r = np.random.Generator(np.random.PCG64(seed + 2))
    return [_u32(r.integers(0, VOCAB, n)) for n, _ in _class_lens(c)]


def _class_prepare(c, seed):
    ctx, lens, toks = _ctx(), _class_lens(c), _class_tokens(c, seed)
    m = _class_model(ctx, c, seed)
    tab, pages = _tables([n for n, _ in lens], seed)
    pool = m.create_pool(pages, len(lens))
    none = np.empty((1, VOCAB), np.float32)
    for i, (n, t) in enumerate(lens):  # what earlier steps have left in the cache
        for a in range(0, n - t, 4096):
            b = min(n - t, a + 4096)
            m.forward_step(pool, _u32(toks[i][a:b]), _u32([b - a]), _u32([b]), _u32(tab[i]),
                           tab.shape[1], _u32([0]), none, _u32([i]))
    s = dict(m=m, pool=pool, B=len(lens), blocks=tab.shape[1], top=max(n for n, _ in lens))
    if c["kind"] == "decode":
        pos = [n - 1 for n, _ in lens]
        slot = [_slots(tab, i, p, p + 1)[0] for i, p in enumerate(pos)]
        s["args"] = [_dev(a) for a in ([t[-1] for t in toks], pos, slot, tab, [n for n, _ in lens])]
        s["logits"] = torch.empty(len(lens), VOCAB, device="cuda")
        return s
    want = _want(c)
    s["host"] = [np.concatenate([x[n - t:] for x, (n, t) in zip(toks, lens)]),
                 _u32([t for _, t in lens]), _u32([n for n, _ in lens]), _u32(tab), tab.shape[1],
                 want, np.empty((len(want), VOCAB), np.float32), _u32(range(len(lens)))]
    return s


def _prompt_run(s):
    s["m"].forward_step(s["pool"], *s["host"])
    return s["host"][6]


def _moe(x, w, q, m, arch):
    z = x @ w[q + "router"].T + (w[q + "router.b"] if arch == "Migurax" else 0)
    if arch == "Revitar":
        share, chosen = torch.topk(torch.softmax(z, -1), m["router"]["top"])
    else:
        best, chosen = torch.topk(z, m["router"]["top"])
        share = torch.softmax(best, -1)
    out = torch.zeros_like(x)
    for e in range(m["router"]["experts"]):
        t, j = torch.nonzero(chosen == e, as_tuple=True)
        h = x[t] @ w[f"{q}e{e}.up"].T
        h = torch.nn.functional.silu(x[t] @ w[f"{q}e{e}.gate"].T) * h if arch == "Revitar" else \
            torch.relu(h) ** 2
        out.index_add_(0, t, share[t, j][:, None] * (h @ w[f"{q}e{e}.down"].T))
    return out


def _sigmoid_attention(x, w, p, m, eps, pos):
    """One layer's mixer on sequences laid end to end; `pos` [(first, end)]."""
    H, G, D = m["heads"], m["kv_heads"], m["dim"]
    q = _rms(x @ w[p + "q"].T, w[p + "q.norm"], eps).view(-1, H, D)
    k = _rms(x @ w[p + "k"].T, w[p + "k.norm"], eps).view(-1, G, D)
    v = (x @ w[p + "v"].T).view(-1, G, D)
    o = torch.zeros_like(q)
    for a, b in pos:
        i = torch.arange(b - a, device="cuda")
        dist = (i[:, None] - i).double()
        seen = (dist >= 0) & (dist < m["mask"]["size"])
        dist = dist.clamp_min(0)
        for h in range(H):
            s = q[a:b, h] @ k[a:b, h * G // H].T * m["scale"]
            s = m["softcap"] * torch.tanh(s / m["softcap"]) + w[p + "pb"][h]
            s = s - w[p + "r1"][h] * torch.log1p(w[p + "r2"][h] * dist)
            o[a:b, h] = torch.where(seen, torch.sigmoid(s), torch.zeros_like(s)) @ \
                v[a:b, h * G // H]
    return o.flatten(1) @ w[p + "o"].T


def _latent(x, w, p, m, eps, pos):
    H, D, RD, DV, R = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
    at = torch.cat([torch.arange(b - a, device="cuda") for a, b in pos]).double()
    angle = at[:, None] * m["rot"]["base"] ** (-torch.arange(0, RD, 2, device="cuda").double() / RD)

    def rot(t):
        g = angle if t.dim() == 2 else angle[:, None]
        u, v = t[..., 0::2], t[..., 1::2]
        return torch.stack([u * g.cos() - v * g.sin(), v * g.cos() + u * g.sin()], -1).flatten(-2)

    q = (_rms(x @ w[p + "dq"].T, w[p + "dq.norm"], eps) @ w[p + "uq"].T).view(-1, H, D + RD)
    down = x @ w[p + "dkv"].T
    lat, kr = _rms(down[:, :R], w[p + "dkv.norm"], eps), rot(down[:, R:])
    qr = rot(q[..., D:])
    k, v = (lat @ w[p + "uk"].T).view(-1, H, D), (lat @ w[p + "uv"].T).view(-1, H, DV)
    o = torch.zeros(x.shape[0], H, DV, dtype=torch.float64, device="cuda")
    for a, b in pos:
        n = b - a
        late = torch.ones(n, n, dtype=torch.bool, device="cuda").triu(1)
        for h in range(H):
            s = (q[a:b, h, :D] @ k[a:b, h].T + qr[a:b, h] @ kr[a:b].T) * m["scale"]
            s = torch.cat([s.masked_fill(late, -math.inf), w[p + "sink"][h].expand(n, 1)], 1)
            o[a:b, h] = torch.softmax(s, -1)[:, :-1] @ v[a:b, h]
    return o.flatten(1) @ w[p + "o"].T


def _memory(x, w, p, m, eps, pos):
    H, D, DV, cap = m["heads"], m["dim"], m["vdim"], m["gate_cap"]
    S, longest = len(pos), max(b - a for a, b in pos)

    def lay(t, *shape):  # [time, sequence, ...], zeros behind each sequence's end
        out = torch.zeros(longest, S, *shape, dtype=torch.float64, device="cuda")
        for i, (a, b) in enumerate(pos):
            out[:b - a, i] = t[a:b].view(b - a, *shape)
        return out

    q, k = lay(x @ w[p + "q"].T * D ** -0.5, H, D), lay(x @ w[p + "k"].T, H, D)
    v = lay(x @ w[p + "v"].T, H, DV)
    gi = lay(cap * torch.tanh((x @ w[p + "i"].T + w[p + "i.b"]) / cap), H)
    gf = lay(torch.nn.functional.logsigmoid(
        cap * torch.tanh((x @ w[p + "f"].T + w[p + "f.b"]) / cap)), H)
    mat = torch.zeros(S, H, D, DV, dtype=torch.float64, device="cuda")
    n, top = torch.zeros_like(k[0]), torch.zeros_like(gi[0])
    o = torch.empty_like(v)
    for t in range(longest):
        new = torch.maximum(gf[t] + top, gi[t])
        keep, take = torch.exp(gf[t] + top - new), torch.exp(gi[t] - new)
        kt = take[..., None] * k[t]
        mat.mul_(keep[..., None, None]).addcmul_(kt[..., None], v[t][..., None, :])
        n, top = keep[..., None] * n + kt, new
        den = torch.maximum((n * q[t]).sum(-1).abs(), torch.exp(-new)) + 1e-6
        o[t] = (q[t][..., None, :] @ mat)[..., 0, :] / den[..., None]
    o = torch.cat([o[:b - a, i] for i, (a, b) in enumerate(pos)])
    o = o / torch.sqrt((o * o).mean(-1, keepdim=True) + eps)
    return o.flatten(1) * w[p + "norm"] * torch.sigmoid(x @ w[p + "g"].T) @ w[p + "o"].T


def _class_exact(c, seed):
    lens, toks = _class_lens(c), _class_tokens(c, seed)
    if sum(n for n, _ in lens) > 40000:
        return None
    cfg, w16 = _class_weights(c, seed)
    ends = np.cumsum([n for n, _ in lens])
    pos = [(int(e) - n, int(e)) for e, (n, _) in zip(ends, lens)]
    eps = cfg["norm"]["eps"]
    x = w16["embed"][torch.from_numpy(np.concatenate(toks).astype(np.int64)).cuda()].double()
    for i, layer in enumerate(cfg["layers"]):
        p = f"l{i}."
        w = {n: t.double() for n, t in w16.items() if n.startswith(p)}
        mix = {"attention": _sigmoid_attention, "latent_attention": _latent, "mlstm": _memory}
        y = mix[layer["type"]](x, w, p + "mix.", layer["mixer"], eps, pos)
        if c["arch"] == "Revitar":
            x = x + cfg["residual_mult"] * _rms(y, w[p + "norm1"], eps)
            y = _moe(x, w, p + "mlp.", layer["mlp"], c["arch"])
            x = x + cfg["residual_mult"] * _rms(y, w[p + "norm2"], eps)
            continue
        x = _rms(cfg["postln_alpha"] * x + y, w[p + "norm1"], eps)
        q = p + "mlp."
        if layer["mlp"]["kind"] == "dense":
            y = torch.relu(x @ w[q + "up"].T + w[q + "up.b"]) ** 2 @ w[q + "down"].T + \
                w[q + "down.b"]
        else:
            y = _moe(x, w, q, layer["mlp"], c["arch"])
        x = _rms(cfg["postln_alpha"] * x + y, w[p + "norm2"], eps)
    rows = torch.cat([torch.arange(e - t, e) for (n, t), e in zip(lens, ends.tolist())]).cuda()
    x = x[rows]
    if c["kind"] == "prompt":
        x = x[torch.from_numpy(_want(c).astype(np.int64)).cuda()]
    x = _rms(x, w16["final.norm"], eps) @ w16["head"].double().T
    return x.cpu().numpy() if c["kind"] == "prompt" else x


def _class_work(c):
    W, H, G, D, win, E, top, F = REVITAR[c["size"]]
    h, d, rd, dv, r, qr, mh, md, mv = MIGURAX[c["size"]]
    lens = _class_lens(c)
    T, L = sum(t for _, t in lens), c["layers"]
    used = E * (1 - (1 - top / E) ** T)  # distinct experts, rows choosing at random
    outs = len(_want(c)) if c["kind"] == "prompt" else T
    byts, flops = 2 * VOCAB * W + 4 * outs * VOCAB, 2 * outs * VOCAB * W
    mats = 3 if c["arch"] == "Revitar" else 2
    for i in range(L):
        dense = c["arch"] == "Migurax" and i == 0
        n = mats * W * F
        byts += 2 * n * (top if dense else used) + (0 if dense else 4 * E * W)
        flops += 2 * T * (n * top + (0 if dense else E * W))
        if c["arch"] == "Revitar":
            n = W * (2 * H * D + 2 * G * D)
            keys = sum(min(win, a - t + j + 1) for a, t in lens for j in range(t))
            byts += 2 * n + 4 * G * D * sum(min(a, win + t) for a, t in lens)
            flops += 2 * T * n + 4 * keys * H * D
        elif i % 2 == 0:
            n, ex = W * (qr + r + rd) + qr * h * (d + rd) + W * h * dv, r * h * (d + dv)
            byts += 2 * (n + ex) + 2 * (r + rd) * sum(a for a, _ in lens)
            flops += 2 * T * n
            for a, t in lens:  # a prompt's latents expanded once, or a decoding row's query
                keys = sum(range(a - t + 1, a + 1))
                flops += 2 * a * ex + 2 * keys * h * (d + rd + dv) if t > 1 else \
                    2 * ex + 2 * keys * h * (2 * r + rd)
        else:
            n = W * (2 * mh * md + 2 * mh * mv + 2 * mh) + W * mh * mv
            byts += 2 * n + 8 * mh * md * mv * len(lens)
            flops += T * (2 * n + 4 * mh * md * mv)
    return dict(bytes=byts, flops=flops)


KINDS = {"ffn": (_ffn_prepare, _ffn_run, _ffn_exact, _ffn_work),
         "chunk": (_chunk_prepare, _chunk_run, _chunk_exact, _chunk_work),
         "llama": (_llama_prepare, _step_run, _llama_exact, _llama_work),
         "prompt": (_class_prepare, _prompt_run, _class_exact, _class_work),
         "decode": (_class_prepare, _step_run, _class_exact, _class_work)}


def prepare(case, seed):
    s = KINDS[case["kind"]][0](case, seed)
    torch.cuda.synchronize()
    s["run"] = KINDS[case["kind"]][1]
    return s


def run(state):
    return state["run"](state)


def exact(case, seed):
    return KINDS[case["kind"]][2](case, seed)


def work(case):
    return KINDS[case["kind"]][3](case)


def tolerance(case):
    """About four times the relative error against float64 that each kind shows, over the range."""
    if case["kind"] == "ffn":
        return {"rel": 2e-3 if case["fmt"] == "q8_0" else 3e-3}
    if case["kind"] == "chunk":
        return {"rel": 2e-4}
    if case["kind"] == "llama":
        return {"rel": 2e-3}
    return {"rel": 3e-2 if case["arch"] == "Revitar" else 2e-2}
