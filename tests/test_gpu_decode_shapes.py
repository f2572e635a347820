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
