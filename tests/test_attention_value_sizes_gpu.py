"""GPU: attention over the quantised pool where V rows differ widely in size: rows near the smallest
and the largest f32 numbers, rows of zeros (stored with the scale 1) among small ones, and a large row
that the softmax all but leaves out. Against float64 over the dequantised pool.

Bounds, of the largest result of a head: 1e-4 for the int8 pool (the query's two planes, 2^-15 of a
head's largest value) and 2e-5 for fp8 (f32 rounding of sums and exponentials); how large the V rows are
takes no part in either.
"""
import numpy as np
import pytest

from cases import dev

pytestmark = pytest.mark.gpu

BS, N, CHUNK = 16, 700, 70


def value_rows(rng, kind, n, width):
    v = rng.standard_normal((n, width)).astype(np.float32)
    if kind == "tiny_first":      # every warp's and every CTA's first tiles
        v[:400] *= np.float32(1e-36)
    elif kind == "tiny_between":
        v[200:500] *= np.float32(1e-36)
    elif kind == "all_tiny":
        v *= np.float32(1e-36)
    elif kind == "huge":
        v *= np.float32(1e34)
    elif kind.startswith("zero_row"):
        v *= np.float32(kind.split()[1])
        v[[5, 40, 333, n - 1]] = 0
        v[333] = -0.0
    elif kind.startswith("quiet_row"):  # its score is far below the others'
        v[[33, 450]] *= 1e3
        v *= np.float32(kind.split()[1])
    return v


KINDS = ["tiny_first", "tiny_between", "all_tiny", "huge", "zero_row 1e-5", "zero_row 1e-7",
         "zero_row 1e-9", "quiet_row 1e-5", "quiet_row 1e-12"]


def setup(ctx, kb, oracle, torch, kind, pool, H, KH, hd, T):
    """A pool of one sequence of N tokens, T query rows, and the rows' float64 results."""
    rng = np.random.Generator(np.random.PCG64(0xB2001100 + H + hd + len(kind)))
    nb = (N + BS - 1) // BS
    blocks = rng.permutation(nb + 3)[:nb].astype(np.uint32)
    slots = (blocks[np.arange(N) // BS] * BS + np.arange(N) % BS).astype(np.uint32)
    base = rng.standard_normal((KH, hd))
    q = (base[None, :, None, :] + 0.3 * rng.standard_normal((T, KH, H // KH, hd)))
    q = q.reshape(T, H * hd).astype(np.float32)
    k = rng.standard_normal((N, KH, hd)) * 0.7
    if kind.startswith("quiet_row"):
        k[[33, 450]] = -5 * base
    k, v = k.reshape(N, KH * hd).astype(np.float32), value_rows(rng, kind, N, KH * hd)
    gp = kb.KvPool(ctx, 1, nb + 3, BS, KH, hd, kb.KV_FP8 if pool == "fp8" else kb.KV_INT8)
    op = oracle.KvPool(1, nb + 3, BS, KH, hd, pool == "fp8")
    assert op.write_slots(0, slots, k, v) == 0
    gp.write_slots(0, dev(torch, slots.astype(np.int32)), dev(torch, k), dev(torch, v), N)
    st, kd, vd = op.gather(0, blocks, N)
    assert st == 0
    kd, vd = (a.astype(np.float64).reshape(N, KH, hd) for a in (kd, vd))
    ref = np.empty((T, H, hd))
    for i in range(T):
        n = N - T + i + 1
        for h in range(H):
            s = kd[:n, h * KH // H] @ q[i, h * hd:(h + 1) * hd].astype(np.float64) * hd ** -0.5
            w = np.exp(s - s.max())
            ref[i, h] = w @ vd[:n, h * KH // H] / w.sum()
    return gp, blocks, q, ref


def check(got, ref, pool):
    bound = 2e-5 if pool == "fp8" else 1e-4
    got = got.reshape(ref.shape).astype(np.float64)
    size = np.abs(ref).max(-1)
    assert size.min() > 0
    err = np.abs(got - ref).max(-1) / size
    assert np.isfinite(err).all() and err.max() <= bound


@pytest.mark.parametrize("H,KH,hd", [(6, 2, 64), (8, 1, 128)])
@pytest.mark.parametrize("pool", ["int8", "fp8"])
@pytest.mark.parametrize("kind", KINDS)
def test_decode(ctx, kb, oracle, torch_cuda, kind, pool, H, KH, hd):
    torch = torch_cuda
    gp, blocks, q, ref = setup(ctx, kb, oracle, torch, kind, pool, H, KH, hd, 1)
    p = kb.PagedAttentionParams(1, H, KH, hd, BS, blocks.size, hd ** -0.5)
    out = torch.full((1, H * hd), float("nan"), device="cuda")
    lens = np.array([N], np.uint32)
    gp.paged_attention(0, dev(torch, q), dev(torch, blocks.astype(np.int32)),
                       dev(torch, lens.astype(np.int32)), out, p, lens)
    ctx.sync()
    check(out.cpu().numpy(), ref, pool)
    gp.destroy()


@pytest.mark.parametrize("H,KH,hd", [(6, 2, 64), (8, 1, 128)])
@pytest.mark.parametrize("pool", ["int8", "fp8"])
@pytest.mark.parametrize("kind", KINDS)
def test_prompt(ctx, kb, oracle, torch_cuda, kind, pool, H, KH, hd):
    torch = torch_cuda
    gp, blocks, q, ref = setup(ctx, kb, oracle, torch, kind, pool, H, KH, hd, CHUNK)
    p = kb.PagedAttentionParams(1, H, KH, hd, BS, blocks.size, hd ** -0.5)
    out = torch.full((CHUNK, H * hd), float("nan"), device="cuda")
    gp.paged_attention_prefill(0, dev(torch, q), dev(torch, blocks.astype(np.int32)),
                               np.array([N], np.uint32), np.array([CHUNK], np.uint32), out, p)
    ctx.sync()
    check(out.cpu().numpy(), ref, pool)
    gp.destroy()
