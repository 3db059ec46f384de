"""GPU: decode attention in tiles of 16 tokens (csrc/paged_decode.cu) against the oracle, at the edges of
its tiles, rings and partitions: contexts of one token, around 16, past a warp's ring and past a
partition, blocks of 16 and of several tiles, every group width's two head tiles.

Tolerances: 1e-4 of the largest result for the int8 pool (the query's two planes: 2^-15 of a head's
largest value) and 2e-5 for fp8 (f32 rounding of sums and exponentials over contexts of thousands).
"""
import numpy as np
import pytest

from cases import permuted_tables
from conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,KH,hd,bs", [(3, 1, 64, 16), (15, 5, 64, 16), (8, 1, 64, 32),
                                        (4, 4, 128, 16), (10, 2, 128, 48), (8, 1, 128, 16)])
@pytest.mark.parametrize("pool", ["int8", "fp8"])
def test_paged_decode_edges(ctx, kb, oracle, torch_cuda, pool, H, KH, hd, bs):
    torch = torch_cuda
    lens = [1, 15, 16, 17, 130, 513, 1100, 2049]
    rng = np.random.Generator(np.random.PCG64(0xB2000D00 + H * 5 + hd + bs))
    NB, tables = permuted_tables(rng, lens, bs)
    tab = np.zeros((len(lens), max(len(t) for t in tables)), np.uint32)
    for i, t in enumerate(tables):
        tab[i, :len(t)], tab[i, len(t):] = t, t[-1]
    typ = kb.KV_FP8 if pool == "fp8" else kb.KV_INT8
    gp = kb.KvPool(ctx, 1, NB, bs, KH, hd, typ)
    op = oracle.KvPool(1, NB, bs, KH, hd, pool == "fp8")
    # every row of the pool holds something, the bytes behind a context's end among them
    for slots, scale in ((np.arange(NB * bs, dtype=np.uint32), 50.0),
                         (np.concatenate([np.asarray(tables[i], np.int64)[np.arange(n) // bs] * bs +
                                          np.arange(n) % bs for i, n in enumerate(lens)])
                          .astype(np.uint32), 1.0)):
        k, v = (scale * rng.standard_normal((slots.size, KH * hd)).astype(np.float32)
                for _ in range(2))
        assert op.write_slots(0, slots, k, v) == 0
        gp.write_slots(0, torch.from_numpy(slots.astype(np.int32)).cuda(), torch.from_numpy(k).cuda(),
                       torch.from_numpy(v).cuda(), slots.size)
    q = rng.standard_normal((len(lens), H * hd)).astype(np.float32)
    hl = np.array(lens, np.uint32)
    p = kb.PagedAttentionParams(len(lens), H, KH, hd, bs, tab.shape[1], hd ** -0.5)
    out = torch.full((len(lens), H * hd), float("nan"), device="cuda")
    gp.paged_attention(0, torch.from_numpy(q).cuda(), torch.from_numpy(tab.astype(np.int32)).cuda(),
                       torch.from_numpy(hl.astype(np.int32)).cuda(), out, p, hl)
    ctx.sync()
    st, ref = oracle.paged_attention_int8(op, 0, q, tab, hl, oracle.PaParams(
        len(lens), H, KH, hd, bs, tab.shape[1], hd ** -0.5))
    assert st == 0
    got = out.cpu().numpy()
    for i in range(len(lens)):
        assert rel_err(got[i], ref[i]) <= (2e-5 if pool == "fp8" else 1e-4), lens[i]


def test_table_of_more_partitions_than_a_grid_holds(ctx, kb, torch_cuda):
    """Without lengths on the host the grid covers the whole table: 65,536 partitions of 2048 tokens are
    more than the grid's third dimension holds, which the general kernel's first does."""
    torch = torch_cuda
    bs, hd, lens = 1024, 64, np.array([37], np.uint32)
    maxb = 65536 * 2048 // bs
    rng = np.random.Generator(np.random.PCG64(0xB2000D80))
    gp = kb.KvPool(ctx, 1, 1, bs, 1, hd, kb.KV_INT8)
    k, v = (torch.from_numpy(rng.standard_normal((37, hd)).astype(np.float32)).cuda()
            for _ in range(2))
    gp.write_slots(0, torch.arange(37, dtype=torch.int32, device="cuda"), k, v, 37)
    q = torch.from_numpy(rng.standard_normal((1, hd)).astype(np.float32)).cuda()
    tab = torch.zeros(maxb, dtype=torch.int32, device="cuda")
    ln = torch.from_numpy(lens.astype(np.int32)).cuda()
    outs = []
    for blocks, host in ((1, lens), (maxb, None)):
        out = torch.full((1, hd), float("nan"), device="cuda")
        gp.paged_attention(0, q, tab, ln, out,
                           kb.PagedAttentionParams(1, 1, 1, hd, bs, blocks, hd ** -0.5), host)
        ctx.sync()
        outs.append(out.cpu().numpy())
    assert rel_err(outs[1], outs[0]) <= 1e-4
    gp.destroy()
