"""The sparse MLP over the forms of its arguments: one call behind both products gives what the two give one by one."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["plain", "int64", "no_bias", "strided_x", "strided_rows", "transposed_w1", "strided_idx", "empty", "wider_out"])
@pytest.mark.parametrize("B", [1, 3, 16])
def test_mlp_sparse_equals_its_two_products(cuda, form, B):
    from dejavu_b200 import ops

    g = torch.Generator(device=cuda).manual_seed(B)
    Z, N, M = 520, 136, 0 if form == "empty" else 77

    def rnd(*shape):
        return torch.randn(*shape, device=cuda, generator=g).mul_(0.1).half()

    x, w1, w2, b1, b2 = rnd(B, N), rnd(Z, N), rnd(Z, N), rnd(Z), rnd(N)
    idx = torch.randperm(Z, device=cuda, generator=g)[:M].int()
    if form == "int64":
        idx = idx.long()
    if form == "no_bias":
        b1 = b2 = None
    if form == "strided_x":
        x = rnd(B, 2 * N)[:, ::2]
    if form == "strided_rows":
        w1, w2 = rnd(Z, N + 8)[:, :N], rnd(Z, N + 16)[:, :N]
    if form == "transposed_w1":
        w1 = rnd(N, Z).t()
    if form == "strided_idx":
        idx = torch.stack([idx, idx], 1)[:, 0]
    if form == "wider_out":
        w2, b2 = rnd(Z, 2 * N), rnd(2 * N)
    want = ops.gather_transposed_gemv(ops.gather_gemv(x, w1, idx, b1, "relu"), w2, idx, b2)
    got = ops.mlp_sparse(x, w1, w2, idx, b1, b2)
    assert got.shape == want.shape and torch.equal(got, want)


@pytest.mark.parametrize("B", [1, 3])
def test_mlp_sparse_takes_weights_with_a_dimension_of_one_behind(cuda, B):
    from dejavu_b200 import ops

    g = torch.Generator(device=cuda).manual_seed(B)
    x, w1, w2 = (torch.randn(n, 136, device=cuda, generator=g).mul_(0.1).half() for n in (B, 520, 520))
    idx = torch.randperm(520, device=cuda, generator=g)[:77]
    assert torch.equal(ops.mlp_sparse(x, w1[..., None], w2[..., None], idx), ops.mlp_sparse(x, w1, w2, idx))


def test_mlp_sparse_refuses_what_its_products_refuse(cuda):
    from dejavu_b200 import ops

    x, w = torch.zeros(2, 64, device=cuda).half(), torch.zeros(128, 64, device=cuda).half()
    idx = torch.arange(4, device=cuda)
    for args in ((x.float(), w, w, idx), (x, w.float(), w, idx), (x, w, w, idx.short()), (x, w, w, idx, w[0]), (x, w, w, idx, None, w[:, 0]),
                 (x.repeat(20, 1), w, w, idx), (x[:, :32], w, w, idx)):
        with pytest.raises(Exception):
            ops.mlp_sparse(*args)
    with pytest.raises(RuntimeError):
        ops.mlp_sparse(x.cpu(), w.cpu(), w.cpu(), idx.cpu())
