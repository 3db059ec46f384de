"""GPU: prompt attention in tiles of query rows (csrc/paged_prefill.cu) at the edges of its tiles of 64
rows and 64 tokens, of the key splits and of a launch's 128 sequences, int8 and fp8 pools, against the
oracle's masked dense attention over the dequantised pool. Bound: the query's two int8 planes are off
by at most amax / (127 * 508) per element, which leaves a few 1e-5 of the output scale; 1e-4 here. The
fp8 form keeps 22 bits of query and weights: 1e-5."""
import numpy as np
import pytest

from cases import dev, permuted_tables
from conftest import rel_err

pytestmark = pytest.mark.gpu

CASES = [  # heads, kv heads, head_dim, block size, [(cached, query tokens)]
    (1, 1, 64, 16, [(0, 3)]),                                  # the fewest tokens a tile takes
    (15, 5, 64, 16, [(63, 64), (0, 65), (1, 21), (129, 22)]),  # both sides of a tile's edges
    (8, 1, 128, 16, [(1000, 8), (0, 9), (513, 70)]),           # group 8, keys in splits
    (6, 2, 128, 8, [(255, 1), (0, 128), (320, 43)]),           # a decoding row among the portions
    (4, 4, 64, 5, [(7, 130), (190, 11)]),                      # pages of an odd size
    (14, 2, 64, 32, [(30, 40), (0, 0), (90, 33)]),             # a sequence without query tokens
    (3, 1, 64, 16, [(2 * i % 37, 1 + i % 9) for i in range(131)]),  # more sequences than a launch
]


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("H,KH,hd,bs,seqs", CASES)
def test_prefill_tiles_match_oracle(ctx, kb, oracle, torch_cuda, H, KH, hd, bs, seqs, fp8):
    torch = torch_cuda
    rng = np.random.Generator(np.random.PCG64(0xB2000F00 + H * 131 + hd + len(seqs)))
    ctx_lens = [max(1, sp + ql) for sp, ql in seqs]
    NB, tables = permuted_tables(rng, ctx_lens, bs)
    maxb = max(len(t) for t in tables)
    gp = kb.KvPool(ctx, 1, NB, bs, KH, hd, kb.KV_FP8 if fp8 else kb.KV_INT8)
    op = oracle.KvPool(1, NB, bs, KH, hd, fp8=fp8)
    padded = np.array([t + [t[-1]] * (maxb - len(t)) for t in tables], np.uint32)
    for s, c in enumerate(ctx_lens):
        t = np.arange(c)
        slots = (np.asarray(tables[s])[t // bs] * bs + t % bs).astype(np.uint32)
        # rows of very different sizes: the scales take part in the softmax's reference
        size = np.exp(rng.uniform(-6, 3, (c, 1))).astype(np.float32)
        k = rng.standard_normal((c, KH * hd), dtype=np.float32)
        v = rng.standard_normal((c, KH * hd), dtype=np.float32) * size
        gp.write_slots(0, dev(torch, slots), dev(torch, k), dev(torch, v), c, slots)
        assert op.write_slots(0, slots, k, v) == 0
    T = sum(ql for _, ql in seqs)
    q = rng.standard_normal((T, H * hd), dtype=np.float32)
    q[T // 2] *= 1e-3  # a flat row
    scale = np.float32(1.0) / np.sqrt(np.float32(hd))
    p = kb.PagedAttentionParams(len(seqs), H, KH, hd, bs, maxb, scale)
    out = torch.full((T, H * hd), float("nan"), dtype=torch.float32, device="cuda")
    args = (dev(torch, q), dev(torch, padded.reshape(-1)), np.array(ctx_lens, np.uint32),
            np.array([ql for _, ql in seqs], np.uint32), out, p)
    gp.paged_attention_prefill(0, *args)
    ctx.sync()
    got = out.cpu().numpy()
    row = 0
    for s, (sp, ql) in enumerate(seqs):
        if ql:
            st, ref = oracle.prefill_attention_int8(op, 0, q[row:row + ql], tables[s], sp, H, scale)
            assert st == 0
            assert rel_err(got[row:row + ql], ref) <= (1e-5 if fp8 else 1e-4), (s, sp, ql)
        row += ql
    # a block id outside the pool is reported, not followed
    bad = padded.copy()
    bad[-1, 0] = NB + 5
    gp.paged_attention_prefill(0, args[0], dev(torch, bad.reshape(-1)), *args[2:])
    with pytest.raises(kb.KansoError) as e:
        ctx.sync()
    assert e.value.code == kb.ERR_SHAPE
    gp.paged_attention_prefill(0, *args)
    ctx.sync()
    assert np.array_equal(out.cpu().numpy(), got)
    gp.destroy()
