"""Decode products at the sizes where their split over blocks can go wrong, against the same product in double."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# Sums of N fp32 products of magnitude ~1 / N, added in some order, are off by at most N rounding errors of 2^-24 of the sum
# of magnitudes and by about sqrt(N) of them in earnest: below 1e-6 of the largest result for every N here, the results'
# own rounding (2^-11 for fp16, 2^-8 for bf16) on top.
ROUNDING = {torch.float32: 2e-6, torch.float16: 2 ** -11 + 2e-6, torch.bfloat16: 2 ** -8 + 2e-6}


def near(got, want):
    err = (got.double() - want).abs().max().item()
    assert err <= ROUNDING[got.dtype] * max(1.0, want.abs().max().item()), err


# rows per block: a fraction, one or two (592 resident blocks), a few, just past a pass of the groups, past a span of 128
@pytest.mark.parametrize("B", [1, 2, 4])
@pytest.mark.parametrize("N,M", [(8, 3), (64, 592), (72, 1185), (1000, 1186), (520, 6000), (2056, 12352), (8, 75777), (16, 160001)])
def test_rows_split_over_resident_blocks(cuda, B, N, M):
    from dejavu_b200 import ops

    g = torch.Generator(device=cuda).manual_seed(B + N + M)
    x = torch.randn(B, N, device=cuda, generator=g).bfloat16()
    w = (torch.randn(M, N, device=cuda, generator=g) * N ** -0.5).bfloat16()
    y = x.double() @ w.double().t()
    near(ops.linear_gemv(x, w, torch.float32), y)
    near(ops.linear_gemv(x, w), y)
    pairs = y[:, :M // 2 * 2]
    gate, up = pairs[:, 0::2], pairs[:, 1::2]
    near(ops.linear_gemv(x, w[:M // 2 * 2], None, "silu_glu"), gate * torch.sigmoid(gate) * up)


@pytest.mark.parametrize("B", [1, 2])
@pytest.mark.parametrize("N,Z,M", [(64, 9, 9), (768, 3072, 384), (136, 5000, 1184), (264, 9000, 4737), (64, 100000, 80003)])
def test_gathered_rows_split_over_resident_blocks(cuda, B, N, Z, M):
    from dejavu_b200 import ops

    g = torch.Generator(device=cuda).manual_seed(B + N + M)
    x = torch.randn(B, N, device=cuda, generator=g).half()
    w = (torch.randn(Z, N, device=cuda, generator=g) * N ** -0.5).half()
    bias = torch.randn(Z, device=cuda, generator=g).half()
    idx = torch.randperm(Z, device=cuda, generator=g)[:M]
    want = (x.double() @ w[idx].double().t() + bias[idx].double()).relu()
    near(ops.gather_gemv(x, w, idx.int(), bias, "relu"), want)
    near(ops.gather_gemv(x, w, idx, bias, "relu"), want)


# the ring: parts of a tile, several tiles, a column tail, one chunk and fewer than a cluster has blocks, 1 to 4 groups of x
@pytest.mark.parametrize("B", [3, 5, 8, 9, 17, 32])
@pytest.mark.parametrize("N,M", [(8, 2), (128, 34), (136, 592), (1000, 1186), (4104, 4096), (2056, 12352), (264, 75778)])
def test_weights_streamed_for_several_rows(cuda, B, N, M):
    from dejavu_b200 import ops

    g = torch.Generator(device=cuda).manual_seed(B + N + M)
    x = torch.randn(B, N, device=cuda, generator=g).bfloat16()
    w = (torch.randn(M, N, device=cuda, generator=g) * N ** -0.5).bfloat16()
    y = x.double() @ w.double().t()
    near(ops.linear_gemv(x, w, torch.float32), y)
    near(ops.linear_gemv(x, w), y)
    gate, up = y[:, 0::2], y[:, 1::2]
    near(ops.linear_gemv(x, w, None, "silu_glu"), gate * torch.sigmoid(gate) * up)
    bias = torch.randn(M, device=cuda, generator=g).half()
    idx = torch.randperm(M, device=cuda, generator=g)[:M - 1]
    want = (x.half().double() @ w.half()[idx].double().t() + bias[idx].double()).relu()
    near(ops.gather_gemv(x.half(), w.half(), idx, bias, "relu"), want)


# rows per block around where the forms of a pass change, fewer rows than warps, a bias that belongs to no row of the first pass
@pytest.mark.parametrize("B", [2, 3, 4])
@pytest.mark.parametrize("N,M", [(8, 1), (768, 385), (2048, 889), (2048, 1481), (2056, 1481), (4096, 593), (4104, 2049), (12288, 445), (3080, 4097)])
def test_few_rows_of_a_few_tokens(cuda, B, N, M):
    from dejavu_b200 import ops

    g = torch.Generator(device=cuda).manual_seed(B + N + M)
    x = torch.randn(B, N, device=cuda, generator=g).half()
    w = (torch.randn(M + 7, N, device=cuda, generator=g) * N ** -0.5).half()
    bias = torch.randn(M + 7, device=cuda, generator=g).half()
    idx = torch.randperm(M + 7, device=cuda, generator=g)[:M]
    y = x.double() @ w.double().t()
    near(ops.gather_gemv(x, w, idx, bias, "relu"), (y + bias.double())[:, idx].relu())
    near(ops.dense_gemv(x, w), y)
    pairs = w[:(M + 7) // 2 * 2].bfloat16()
    p = x.bfloat16().double() @ pairs.double().t()
    near(ops.linear_gemv(x.bfloat16(), pairs, None, "silu_glu"), p[:, 0::2] * torch.sigmoid(p[:, 0::2]) * p[:, 1::2])


# both sides of the line between the form without a ring and the ring; parts of a tile, of a 32-column block, of a split
@pytest.mark.parametrize("B", [5, 8, 9, 16, 17, 25, 32])
@pytest.mark.parametrize("N,M", [(8, 1), (40, 17), (512, 2048), (520, 257), (1024, 4096), (1032, 513), (2048, 1026), (4096, 2048), (4104, 512),
                                 (264, 11265), (12288, 33)])
def test_short_lists_of_several_tokens(cuda, B, N, M):
    from dejavu_b200 import ops

    g = torch.Generator(device=cuda).manual_seed(B + N + M)
    x = torch.randn(B, N, device=cuda, generator=g).half()
    w = (torch.randn(M + 5, N, device=cuda, generator=g) * N ** -0.5).half()
    bias = torch.randn(M + 5, device=cuda, generator=g).half()
    idx = torch.randperm(M + 5, device=cuda, generator=g)[:M]
    near(ops.gather_gemv(x, w, idx.int(), bias, "relu"), (x.double() @ w[idx].double().t() + bias[idx].double()).relu())
    pairs = w[:(M + 1) // 2 * 2].bfloat16()
    p = x.bfloat16().double() @ pairs.double().t()
    near(ops.linear_gemv(x.bfloat16(), pairs, torch.float32), p)
    near(ops.linear_gemv(x.bfloat16(), pairs, None, "silu_glu"), p[:, 0::2] * torch.sigmoid(p[:, 0::2]) * p[:, 1::2])


@pytest.mark.parametrize("B,E,top,D,F,Fs", [(2, 1, 1, 8, 8, 0), (3, 5, 2, 136, 24, 40), (8, 8, 2, 512, 200, 328), (9, 40, 3, 264, 136, 8),
                                            (17, 4, 4, 1032, 72, 0), (32, 300, 1, 64, 16, 16), (24, 60, 5, 136, 64, 8),
                                            (8, 130, 16, 264, 40, 0), (31, 1137, 16, 64, 8, 0), (2, 33, 15, 64, 24, 16)])
def test_routed_weights_streamed_for_several_rows(cuda, B, E, top, D, F, Fs):
    from dejavu_b200 import ops

    g = torch.Generator(device=cuda).manual_seed(B + E + D)

    def rnd(*shape):
        return torch.randn(*shape, device=cuda, generator=g).mul_(shape[-1] ** -0.5).bfloat16()

    x, z = torch.randn(B, D, device=cuda, generator=g).bfloat16(), torch.randn(B, E, device=cuda, generator=g)
    gu, down = rnd(E, 2 * F, D), rnd(E, D, F)
    shared = (rnd(2 * Fs, D), rnd(D, Fs)) if Fs else (None, None)
    got = ops.moe_decode(x, z, gu, down, top, *shared)

    def unit(v, up, dn):  # the activation is kept in bf16, as it was before
        p = v @ up.double().t()
        a = p[:, 0::2] * torch.sigmoid(p[:, 0::2]) * p[:, 1::2]
        return a.bfloat16().double() @ dn.double().t()

    want = unit(x.double(), *shared) if Fs else torch.zeros(B, D, dtype=torch.float64, device=cuda)
    w, idx = torch.sigmoid(z.double()).topk(top, 1)
    for b in range(B):
        for k in range(top):
            want[b] += unit(w[b, k] * x[b:b + 1].double(), gu[idx[b, k]], down[idx[b, k]])[0]
    # an activation on the edge of two bf16 values may round the other way: 2^-8 of itself, among F * (top + 1) that add up
    assert (got.double() - want).norm() <= 2e-3 * want.norm()


# one row: fewer outputs than blocks, a block's outputs on both sides of a pass and of what it keeps, experts of few and of many chunks
@pytest.mark.parametrize("E,top,D,F,Fs", [(1, 1, 8, 8, 0), (5, 2, 136, 24, 40), (8, 2, 2048, 1856, 1856), (40, 16, 264, 136, 8), (4, 4, 1032, 72, 0),
                                          (300, 1, 64, 16, 20000), (3, 2, 40, 30008, 0), (1024, 3, 8, 8, 16), (2, 2, 9224, 600, 328), (4, 1, 76000, 16, 8)])
def test_routed_weights_of_one_row(cuda, E, top, D, F, Fs):
    test_routed_weights_streamed_for_several_rows(cuda, 1, E, top, D, F, Fs)


# Distance of fp32 results from 64 bits. An addition rounds by about 2.4e-8 of the sum so far (2^-23 / sqrt(12), averaged over the
# mantissa), which grows evenly: n in a row are off by 2.4e-8 * sqrt(n / 2) of the result, and the warps' and blocks' sums add 8
# more; the products of an MMA that starts from zero are cut by 6e-8 to 7e-8. With 3 and 4 rows parts of 8 additions are joined,
# up to 8 rows add every 16 columns of a warp's quarter, more rows every 32. Sums left in the tensor cores' accumulators are 1e-6
# off at 4096 columns and 3e-6 at 11008.
@pytest.mark.parametrize("B", [3, 4, 5, 8, 17, 32])
@pytest.mark.parametrize("N,M", [(768, 50272), (2560, 8192), (4096, 4096), (4096, 22016), (11008, 8192)])
def test_sums_of_several_rows_are_fp32_sums(cuda, B, N, M):
    from dejavu_b200 import ops

    g = torch.Generator(device=cuda).manual_seed(B + N)
    x = torch.randn(B, N, device=cuda, generator=g).bfloat16()
    w = (torch.randn(M, N, device=cuda, generator=g) * N ** -0.5).bfloat16()
    y = x.double() @ w.double().t()
    n = 8 + N / 512 if B <= 4 else N / 64 if B <= 8 else N / 128
    assert (ops.linear_gemv(x, w, torch.float32).double() - y).norm() <= (2.4e-8 * (n / 2 + 8) ** 0.5 + 7e-8) * y.norm()
