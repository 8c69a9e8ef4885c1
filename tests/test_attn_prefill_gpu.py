"""Attention of prompt rows on tcgen05 (attn_prefill.cu): both kinds of cache against a plain float64 statement, at the edges of its tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
D = 128


@pytest.fixture(scope="module")
def ops():
    from libtbvcoll_b200 import ops as o
    return o


def rnd(*shape, seed, scale=1.0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return (torch.randn(shape, generator=g, device=DEV) * scale).to(torch.bfloat16)


def plain(q, k, v, scale, see, first, cap=0.0):
    """q [T, H, D], k / v [n, G, D]; row t sees keys first[t] .. see[t] - 1.  Returns the result and the same sum over |v|, which bounds what rounding can do."""
    T, H = q.shape[:2]
    rep = H // k.shape[1]
    q, k, v = q.double(), k.double().repeat_interleave(rep, 1), v.double().repeat_interleave(rep, 1)
    s = torch.einsum("ihd,jhd->hij", q, k) * scale
    if cap:
        s = cap * torch.tanh(s / cap)
    j = torch.arange(k.shape[0], device=DEV)[None]
    s = s.masked_fill((j >= see[:, None]) | (j < first[:, None]), float("-inf"))
    p = torch.softmax(s, -1)
    return torch.einsum("hij,jhd->ihd", p, v), torch.einsum("hij,jhd->ihd", p, v.abs())


def check(got, want, size):
    # bf16 has 8 significant bits: weights rounded by up to 2^-8 of each, the result by 2^-8, together 2^-7 of the sum over |v|; fp32 sums, scores (below 2^5: they move a
    # weight by 2^-18) and the approximate exponential are far below
    assert torch.isfinite(got).all()
    assert ((got.double() - want).abs() <= size * 2.0 ** -6.95 + 1e-6).all()


def layout(lens, starts, bs, seed):
    """Block tables over shuffled blocks; rows beyond a sequence's last token hold NaN patterns in the caches made by the tests."""
    need = [(s + n + bs - 1) // bs for n, s in zip(lens, starts)]
    perm = torch.randperm(sum(need) + 3, generator=torch.Generator().manual_seed(seed)) + 0
    tables, at = torch.zeros(len(lens), max(need) + 1, dtype=torch.int32), 0
    for i, n in enumerate(need):
        tables[i, :n] = perm[at: at + n].to(torch.int32)
        at += n
    return tables, sum(need) + 3


LENS, STARTS = [129, 1, 31, 128, 300, 33], [0, 127, 128, 129, 5, 700]


# keys: what the caller says of the longest context (64 or less: the 64-row form); off: channels by which the results lie beside a 32-byte boundary (rows then are no multiple of 32 bytes either)
@pytest.mark.parametrize("nq,nkv,bs,tile_rows,off,keys", [(8, 2, 16, 128, 0, 0), (8, 2, 16, 64, 0, 0), (4, 4, 48, 128, 0, 0), (8, 1, 32, 128, 0, 64), (4, 2, 16, 100, 0, 64), (8, 2, 16, 128, 8, 0), (4, 4, 16, 64, 8, 0),
                                                     (8, 2, 16, 64, 4, 0), (8, 2, 8, 64, 0, 0), (4, 4, 24, 64, 2, 0), (8, 1, 8, 64, 0, 0), (4, 2, 40, 64, 0, 0),
                                                          (8, 2, 16, 64, 0, 64), (4, 4, 48, 64, 0, 1), (8, 2, 16, 64, 0, 65)])
def test_split_caches(ops, nq, nkv, bs, tile_rows, off, keys):
    tables, nblocks = layout(LENS, STARTS, bs, 1)
    kc, vc = rnd(nblocks * bs, nkv, D, seed=1), rnd(nblocks * bs, nkv, D, seed=2)
    written = torch.zeros(nblocks * bs, dtype=torch.bool)
    slots = []
    for i, (n, s) in enumerate(zip(LENS, STARTS)):
        pos = torch.arange(n + s)
        slots.append(tables[i, pos // bs].long() * bs + pos % bs)
        written[slots[-1]] = True
    kc[~written.to(DEV)] = float("nan")                     # what nobody wrote must not matter
    vc[~written.to(DEV)] = float("nan")
    seqof = torch.tensor(sum(([i] * n for i, n in enumerate(LENS)), []), dtype=torch.int32)
    ctx = torch.tensor(sum(([s + t + 1 for t in range(n)] for n, s in zip(LENS, STARTS)), []), dtype=torch.int32)
    T, scale = int(seqof.numel()), 0.2
    wide = rnd(T, (nq + 2 * nkv) * D, seed=3)
    q = wide.view(T, -1, D)[:, :nq]                          # as in the model: a view into the projection
    around = torch.full((T, nq * D + off), 7.0, dtype=torch.bfloat16, device=DEV)
    out = around[:, off:].unflatten(1, (nq, D))
    tiles = ops.prefill_tiles(seqof, nq // nkv, tile_rows)
    assert ops.prefill_tile_rows(bs) == (64 if bs % 16 else 128)
    ops.prefill_attention(q, kc, vc, tables.to(DEV), ctx.to(DEV), seqof.to(DEV), tiles.to(DEV), out, scale, bs, tile_rows, keys)
    torch.cuda.synchronize()
    assert not ops.gemm_error()
    r0 = 0
    for i, (n, s) in enumerate(zip(LENS, STARTS)):
        rows = slots[i].to(DEV)
        see = torch.arange(s + 1, s + n + 1, device=DEV)
        check(out[r0: r0 + n], *plain(q[r0: r0 + n], kc[rows], vc[rows], scale, see, torch.zeros_like(see)))
        r0 += n
    assert (around[:, :off] == 7).all()


# both CTAs of a cluster at work on a unit: one tile of keys (nothing for the second CTA), the edges of two and three, contexts before the prompt; 37 and 38
# tiles of 4 key heads are the last grid that is shared out on 148 SMs and the first that is not.  The stated longest context only chooses the kernel.
@pytest.mark.parametrize("nq,nkv,rows,before", [(4, 1, 1, 0), (4, 1, 128, 0), (4, 1, 129, 0), (8, 2, 256, 0), (8, 2, 257, 0), (8, 1, 40, 345), (4, 4, 385, 127), (16, 4, 1184, 0), (16, 4, 1216, 0)])
def test_keys_shared_out_over_two_ctas(ops, nq, nkv, rows, before):
    n, bs = rows + before, 16
    q, kc, vc = rnd(rows, nq, D, seed=8), rnd(n + 16, nkv, D, seed=9), rnd(n + 16, nkv, D, seed=10)
    kc[n:], vc[n:] = float("nan"), float("nan")
    tables = torch.arange(n // bs + 1, dtype=torch.int32)[None].to(DEV)
    see = torch.arange(before + 1, n + 1, device=DEV)
    seq = torch.zeros(rows, dtype=torch.int32)
    tiles = ops.prefill_tiles(seq, nq // nkv, 128).to(DEV)
    out = torch.full_like(q, float("nan"))
    ops.prefill_attention(q, kc, vc, tables, see.to(torch.int32), seq.to(DEV), tiles, out, 0.2, bs, 128, 2000)
    torch.cuda.synchronize()
    assert not ops.gemm_error()
    check(out, *plain(q, kc[:n], vc[:n], 0.2, see, torch.zeros_like(see)))


def test_growing_and_huge_scores(ops):
    """Keys whose scores grow by more than the rescaling threshold from tile to tile, fall again, and single keys that take all of the weight."""
    n, bs = 700, 16
    q, kc, vc = rnd(n, 4, D, seed=5), rnd(n + 16, 1, D, seed=6), rnd(n + 16, 1, D, seed=7)
    size = torch.ones(n + 16, device=DEV)
    size[128:256], size[256:384], size[500], size[640:] = 3.0, 0.01, 20.0, 6.0
    kc = (kc.float() * size[:, None, None]).to(torch.bfloat16)
    tables = torch.arange(n // bs + 1, dtype=torch.int32)[None].to(DEV)
    see = torch.arange(1, n + 1, device=DEV)
    seq = torch.zeros(n, dtype=torch.int32)
    out = torch.empty_like(q)
    ops.prefill_attention(q, kc, vc, tables, see.to(torch.int32), seq.to(DEV), ops.prefill_tiles(seq, 4, 128).to(DEV), out, 0.3, bs, 128)
    want, size = plain(q, kc[:n], vc[:n], 0.3, see, torch.zeros_like(see))
    assert torch.isfinite(out).all() and not ops.gemm_error()
    # scores reach 2^9: their 24 bits (and the product with the scale) move a weight by up to 2^-12
    assert ((out.double() - want).abs() <= size * 2.0 ** -6.8 + 1e-6).all()


@pytest.mark.parametrize("H,G,window,chunk,cap,gated,bs,off", [(8, 2, 0, 0, 0.0, False, 16, 0), (4, 4, 130, 0, 0.0, True, 16, 0), (8, 1, 0, 200, 20.0, False, 16, 0),
                                                               (12, 2, 1, 0, 50.0, True, 16, 0), (20, 1, 128, 0, 0.0, False, 16, 0), (8, 2, 130, 0, 0.0, True, 16, 8),
                                                               (8, 2, 0, 0, 0.0, True, 8, 0), (12, 2, 130, 0, 50.0, False, 24, 8), (4, 4, 0, 200, 0.0, False, 8, 0)])
def test_paired_rows(ops, H, G, window, chunk, cap, gated, bs, off):
    tables, nblocks = layout(LENS, STARTS, bs, 2)
    row = 2 * D + 8
    cache = rnd(nblocks * G * bs, row, seed=11)
    at = []
    written = torch.zeros(nblocks * G * bs, dtype=torch.bool)
    for i, (n, s) in enumerate(zip(LENS, STARTS)):
        pos = torch.arange(n + s)
        at.append(((tables[i, pos // bs].long() * G)[:, None] + torch.arange(G)[None]) * bs + (pos % bs)[:, None])        # [tokens, G]
        written[at[-1].reshape(-1)] = True
    cache[~written.to(DEV)] = float("nan")
    seqof = torch.tensor(sum(([i] * n for i, n in enumerate(LENS)), []), dtype=torch.int32)
    T = int(seqof.numel())
    q, gate = rnd(T, H * D + 64, seed=12, scale=0.3), rnd(T, H * D, seed=13)
    tiles, r0 = [], 0
    for n, s in zip(LENS, STARTS):
        tiles += [(r0 + k, min(64, n - k), 0, s + k + 1) for k in range(0, n, 64)]
        r0 += n
    tiles = torch.tensor(tiles, dtype=torch.int32, device=DEV)
    around = torch.full((T, H * D + off), 7.0, dtype=torch.bfloat16, device=DEV)
    out = around[:, off:]
    ops.paired_attention_prefill(q, cache, tables.to(DEV), seqof.to(DEV), tiles, out, H, G, D, bs, cap, window, chunk, gate if gated else None)
    torch.cuda.synchronize()
    assert not ops.gemm_error()
    r0 = 0
    for i, (n, s) in enumerate(zip(LENS, STARTS)):
        kv = cache[at[i].to(DEV)]                             # [tokens, G, row]
        see = torch.arange(s + 1, s + n + 1, device=DEV)
        first = (see - window).clamp(min=0) if window else (see - 1) // chunk * chunk if chunk else torch.zeros_like(see)
        want, size = plain(q[r0: r0 + n, : H * D].view(n, H, D), kv[..., :D], kv[..., D: 2 * D], 1.0, see, first, cap)
        if gated:
            f = torch.sigmoid(gate[r0: r0 + n].double()).view(n, H, D)
            want, size = want * f, size * f
        check(out[r0: r0 + n].unflatten(1, (H, D)), want, size)
        r0 += n
    assert (around[:, :off] == 7).all()


@pytest.mark.parametrize("paired,hpk", [(False, 4), (False, 1), (True, 4), (True, 6)])
def test_a_rows_bits_are_its_own(ops, paired, hpk):
    """The bits of a row depend on its own query, keys and values: not on the rows of the next sequence that the same MMA holds, not on a neighbour whose scores grow from
    tile to tile, and not on what an earlier kernel left in the rows of shared memory that no query fills (128 is no multiple of six heads)."""
    bs, G, start, n = 16, 2, 500, 13
    H, keys = G * hpk, start + n + 3
    k, v = rnd(keys // bs * bs + bs, G, D, seed=21), rnd(keys // bs * bs + bs, G, D, seed=22)
    k = (k.float() * (1 + torch.arange(k.shape[0], device=DEV) // 128)[:, None, None]).to(torch.bfloat16)
    cache = torch.zeros(k.shape[0] // bs, G, bs, 2 * D + 8, dtype=torch.bfloat16, device=DEV)
    cache[..., :D], cache[..., D: 2 * D] = k.view(-1, bs, G, D).transpose(1, 2), v.view(-1, bs, G, D).transpose(1, 2)
    cache = cache.view(-1, 2 * D + 8)

    def run(q, counts, heads=H):
        T = q.shape[0]
        tables = torch.arange(k.shape[0] // bs, dtype=torch.int32, device=DEV)[None].expand(len(counts), -1).contiguous()
        seq = torch.tensor(sum(([i] * c for i, c in enumerate(counts)), []), dtype=torch.int32)
        out = torch.empty(T, heads * D, dtype=torch.bfloat16, device=DEV)
        if paired:
            tiles = [(sum(counts[:i]) + a, min(64, c - a), 0, start + a + 1) for i, c in enumerate(counts) for a in range(0, c, 64)]
            ops.paired_attention_prefill(q, cache, tables, seq.to(DEV), torch.tensor(tiles, dtype=torch.int32, device=DEV), out, heads, G, D, bs, 0.0, 0, 0, None)
        else:
            see = torch.cat([torch.arange(start + 1, start + c + 1) for c in counts]).to(torch.int32).to(DEV)
            tiles = ops.prefill_tiles(seq, heads // G, 128).to(DEV)
            ops.prefill_attention(q.view(T, heads, D), k, v, tables, see, seq.to(DEV), tiles, out.view(T, heads, D), 1.0, bs, 128)
        torch.cuda.synchronize()
        return out.view(T, heads, D)

    def dirty(size):                       # leaves queries of this size in shared memory of every SM
        run(rnd(6400, 8 * D, seed=23, scale=size), [13] * 492 + [4], heads=8)

    q = rnd(n, H * D, seed=24, scale=0.1)
    dirty(0.0)
    alone = run(q, [n])
    assert torch.isfinite(alone).all()
    beside = run(torch.cat((q, rnd(40, H * D, seed=25, scale=30.0))), [n, 40])
    assert torch.equal(beside[:n], alone)
    other = q.clone()
    other[5, :D] *= 300.0
    got = run(other, [n])
    got[5, 0] = alone[5, 0]
    assert torch.equal(got, alone)
    dirty(30.0)
    assert torch.equal(run(q, [n]), alone)
