"""A norm folded into the products around it (``gemm_resid``, ``gemm_scaled``, ``gemm_qkv_rope(sq=)``): every form, tile and share of K against the same in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV, EPS = "cuda:0", 1e-5


def rnd(*shape, seed, scale=1.0):
    return (torch.randn(shape, generator=torch.Generator(device=DEV).manual_seed(seed), device=DEV) * scale).to(torch.bfloat16)


# rows of the decode form (its K shared out over clusters, then not) and of the many-token forms; hidden sizes that leave half of a 256-feature tile
@pytest.mark.parametrize("mode", [1, 2, 3, 4])
@pytest.mark.parametrize("T", [1, 5, 64, 200, 383, 384, 513, 1100])
@pytest.mark.parametrize("H,K", [(128, 64), (384, 1096), (2048, 520)])
def test_product_residual_gain_and_squares(mode, T, H, K):
    from libtbvcoll_b200 import ops
    x, w, h0, gain = rnd(T, K, seed=1), rnd(H, K, seed=2, scale=K ** -0.5), rnd(T, H, seed=3), rnd(H, seed=4)
    h, out, sq = h0.clone(), torch.zeros(T, H, dtype=torch.bfloat16, device=DEV), ops.RowSquares(T, H, DEV)
    ops.gemm_persist_mode(mode)
    try:
        ops.gemm_resid(x, w, h, gain, out, sq)
        torch.cuda.synchronize()
    finally:
        ops.gemm_persist_mode(None)
    assert not ops.gemm_error()
    want = h0.double() + x.double() @ w.double().t()
    sums = (x.double().abs() @ w.double().abs().t()) * K * 2.0 ** -24                  # K fp32 additions
    assert ((h.double() - want).abs() <= want.abs() * 2.0 ** -8 + sums).all()          # and one rounding to bf16
    assert torch.equal(out, (h.float() * gain.float()).to(torch.bfloat16))
    got = sq.sums[: sq.parts * sq.ld].view(sq.parts, sq.ld).double().sum(0)[:T]
    assert ((got - h.double().pow(2).sum(1)).abs() <= h.double().pow(2).sum(1) * H * 2.0 ** -24).all()


def squares_of(h, parts, T):
    """Squares of the rows of h by `parts` equal parts of a row, in a buffer of larger stride."""
    from libtbvcoll_b200 import ops
    sq = ops.RowSquares(T, h.shape[1], DEV)
    sq.left_by(parts, T + 3)
    sq.sums[: parts * (T + 3)].view(parts, T + 3)[:, :T] = h.float().pow(2).view(T, parts, -1).sum(2).t()
    return sq


@pytest.mark.parametrize("mode", [1, 2, 3, 4])
@pytest.mark.parametrize("T,parts", [(1, 1), (1, 64), (5, 8), (64, 3), (130, 64), (200, 4), (384, 16), (700, 24)])
@pytest.mark.parametrize("M,K", [(256, 768), (1040, 384)])
def test_products_behind_the_norm(mode, T, parts, M, K):
    from libtbvcoll_b200 import ops
    h, gain, w = rnd(T, K, seed=1, scale=3.0), rnd(K, seed=2), rnd(M, K, seed=3, scale=K ** -0.5)
    x, sq = (h.float() * gain.float()).to(torch.bfloat16), squares_of(h, parts, T)
    scale = (h.double().pow(2).mean(1, keepdim=True) + EPS).rsqrt()
    want = (x.double() @ w.double().t()) * scale
    e = (x.double().abs() @ w.double().abs().t()) * scale * (K + 8) * 2.0 ** -24
    pick = torch.randperm(T, generator=torch.Generator().manual_seed(5))[: max(1, T // 2)].to(DEV)
    got, act, some = (torch.zeros(n, m, dtype=torch.bfloat16, device=DEV) for n, m in ((T, M), (T, M // 2), (pick.numel(), M)))
    ops.gemm_persist_mode(mode)
    try:
        ops.gemm_scaled(x, w, got, sq, EPS)
        ops.gemm_scaled(x, w, act, sq, EPS, epi=ops.EPI_SILU_MUL)
        ops.gemm_scaled(x[pick].contiguous(), w, some, sq, EPS, rows=pick)
        torch.cuda.synchronize()
    finally:
        ops.gemm_persist_mode(None)
    assert not ops.gemm_error()
    assert ((got.double() - want).abs() <= want.abs() * 2.0 ** -8 + e).all()
    assert ((some.double() - want[pick]).abs() <= want[pick].abs() * 2.0 ** -8 + e[pick]).all()
    g, u, ge, ue = want[:, 0::2], want[:, 1::2], e[:, 0::2], e[:, 1::2]
    silu = g * torch.sigmoid(g)
    # roundings of gate, silu and up to bf16 and the result's; the slope of silu is at most 1.1
    assert ((act.double() - silu * u).abs() <= (silu * u).abs() * 2.0 ** -6 + 1.1 * (ge + g.abs() * 2.0 ** -8) * u.abs() + silu.abs() * ue + 1e-6).all()


@pytest.mark.parametrize("mode", [1, 2, 3, 4])
@pytest.mark.parametrize("T,nq,nkv,K", [(1, 4, 2, 512), (17, 16, 4, 2048), (300, 3, 1, 256), (401, 3, 1, 1000), (1025, 8, 4, 256)])
def test_qkv_projection_behind_the_norm(mode, T, nq, nkv, K):
    """With scales that are powers of two: the plain projection of rows scaled before it."""
    from libtbvcoll_b200 import ops
    D, M = 128, (nq + 2 * nkv) * 128
    x, w, b = rnd(T, K, seed=1), rnd(M, K, seed=2, scale=0.05), rnd(M, seed=3)
    pos, cs = (torch.arange(T, dtype=torch.int32) % 250).to(DEV), ops.rope_cos_sin(D, 256, 5e5, DEV)
    slots = torch.arange(T, device=DEV)
    sq = ops.RowSquares(T, K, DEV)
    ratio = 2.0 ** (torch.arange(T, device=DEV) % 5 - 2).float()
    sq.sums[:T] = K / ratio.pow(2)                    # 1 / rms = ratio, but for last places of the mean and the square root
    sq.left_by(1, T)
    got, want = ([torch.zeros(T, M, dtype=torch.bfloat16, device=DEV)] + [torch.zeros(T, nkv, D, dtype=torch.bfloat16, device=DEV) for _ in range(2)] for _ in range(2))
    ops.gemm_persist_mode(mode)
    try:
        ops.gemm_qkv_rope(x, w, got[0], pos, cs, slots, got[1], got[2], nq, nkv, bias=b, sq=sq, eps=0.0)
        ops.gemm_qkv_rope((x.float() * ratio[:, None]).to(torch.bfloat16), w, want[0], pos, cs, slots, want[1], want[2], nq, nkv, bias=b)
        torch.cuda.synchronize()
    finally:
        ops.gemm_persist_mode(None)
    assert not ops.gemm_error()
    for a, c in zip(got, want):
        # a scale off by a last place may turn the roundings of a sum, of its products with cos and sin and of the result, each of 2^-8
        assert ((a.double() - c.double()).abs() <= 4 * 2.0 ** -8 * c.double().abs().amax(-1, keepdim=True)).all() and (a != c).double().mean() < 0.02


def test_embedding_with_the_first_gain():
    from libtbvcoll_b200 import ops
    table, gain = rnd(100, 1032, seed=1), rnd(1032, seed=2)
    ids = torch.tensor([3, 99, 0, 100, -1], device=DEV)
    h, y, sq = torch.empty(5, 1032, dtype=torch.bfloat16, device=DEV), torch.empty(5, 1032, dtype=torch.bfloat16, device=DEV), ops.RowSquares(5, 1032, DEV)
    ops.embed_gain(ids, table, gain, h, y, sq)
    want = torch.cat((table[[3, 99, 0]], torch.zeros(2, 1032, dtype=torch.bfloat16, device=DEV)))
    assert torch.equal(h, want) and torch.equal(y, (want.float() * gain.float()).to(torch.bfloat16))
    assert ((sq.sums[:5].double() - want.double().pow(2).sum(1)).abs() <= want.double().pow(2).sum(1) * 1032 * 2.0 ** -24).all()
