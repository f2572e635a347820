"""The projections of a decode step of several sequences with one lazy-K/V state, against the same products in double."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# one rounding to fp16 behind fp32 sums (see test_gpu_decode_shapes)
ROUNDING = 2 ** -11 + 2e-6


def near(got, want):
    err = (got.double() - want).abs().max().item()
    assert err <= ROUNDING * max(1.0, want.abs().max().item()), err


# token rows per pass (1 .. 64) and passes, columns that end inside a stage, fewer columns than a cluster has blocks
@pytest.mark.parametrize("B,nheads,hd,d", [(2, 5, 32, 8), (3, 4, 64, 328), (5, 32, 128, 4096), (9, 3, 128, 1000), (16, 12, 64, 768),
                                           (17, 2, 32, 72), (33, 2, 128, 136), (2, 12, 128, 768), (2, 30, 32, 72), (3, 12, 64, 2056),
                                           (3, 9, 128, 4104), (47, 3, 64, 136)])
def test_lazy_projection_of_a_batch(cuda, B, nheads, hd, d):
    from dejavu_b200 import _lib, ops

    g = torch.Generator(device=cuda).manual_seed(B + d)
    prompt, steps = 5, 35
    S = prompt + steps
    w = (torch.randn(3, nheads, hd, d, device=cuda, generator=g) * d ** -0.5).half()
    bias = torch.randn(3, nheads, hd, device=cuda, generator=g).half()
    f16 = {"dtype": torch.float16, "device": cuda}
    ring, q = torch.zeros(B, 16, d, **f16), torch.zeros(B, nheads, hd, **f16)
    k, v = torch.zeros(B, nheads, hd // 8, S, 8, **f16), torch.zeros(B, nheads, S, hd, **f16)
    want_k, want_v = (torch.zeros(B, nheads, S, hd, dtype=torch.float64, device=cuda) for _ in range(2))
    state = torch.zeros(_lib.ATTN_STATE_HDR + 3 * nheads, dtype=torch.int32, device=cuda)
    _lib.call("djv_attn_state_reset", state.data_ptr(), nheads, prompt, ops._stream())
    waiting = [[] for _ in range(nheads)]  # (position, token rows) that a head has not seen
    for t in range(steps):
        x = torch.randn(B, d, device=cuda, generator=g).half()
        few = torch.randperm(nheads, device=cuda, generator=g)[:max(1, nheads // 3)].int()
        _lib.call("djv_attn_step_project_batch", q.data_ptr(), w.data_ptr(), bias.data_ptr(), x.data_ptr(), ring.data_ptr(),
                  k.data_ptr(), v.data_ptr(), state.data_ptr(), few.data_ptr(), few.numel(), d, nheads, hd, S, B, ops._stream())
        full = torch.einsum("bd,chjd->cbhj", x.double(), w.double()) + bias.double()[:, None]
        heads = range(nheads) if t % 16 == 15 else few.tolist()
        for h in range(nheads):
            waiting[h].append((prompt + t, full[1:, :, h]))
        for h in heads:
            for pos, kv in waiting[h]:
                want_k[:, h, pos], want_v[:, h, pos] = kv[0], kv[1]
            waiting[h] = []
        used = torch.tensor(sorted(heads), device=cuda)
        near(q[:, used], full[0][:, used])
        near(k.transpose(2, 3).reshape(B, nheads, S, hd), want_k)
        near(v, want_v)
        assert torch.equal(ring[:, t % 16], x)
    assert state[3].item() == 0


# qkv_sparse_kernel (two and three sequences, one row per block where d or hd leave few) and qkv_batch_kernel
@pytest.mark.parametrize("B,nheads,hd,d,nnz", [(2, 30, 32, 72, 12), (3, 32, 128, 4096, 12), (9, 40, 128, 264, 33), (2, 4, 64, 136, 1), (17, 3, 32, 72, 3)])
def test_step_opened_by_the_selection_of_heads(cuda, B, nheads, hd, d, nnz):
    """The selection opens the step and the projection stashes the tokens: the same bits as with a launch that does both first."""
    from dejavu_b200 import _lib, ops

    g = torch.Generator(device=cuda).manual_seed(B + d)
    S, f16 = 40, {"dtype": torch.float16, "device": cuda}
    w, bias = (torch.randn(3, nheads, hd, d, device=cuda, generator=g) * d ** -0.5).half(), torch.randn(3, nheads, hd, generator=g, **f16)
    sides = [(torch.zeros(B, nheads, hd, **f16), torch.zeros(B, 16, d, **f16), torch.zeros(B, nheads, hd // 8, S, 8, **f16),
              torch.zeros(B, nheads, S, hd, **f16), torch.zeros(_lib.ATTN_STATE_HDR + 3 * nheads, dtype=torch.int32, device=cuda)) for _ in range(2)]
    for side in sides:
        _lib.call("djv_attn_state_reset", side[4].data_ptr(), nheads, 3, ops._stream())
    for t in range(35):
        x = torch.randn(B, d, device=cuda, generator=g).half()
        scores = torch.randn(nheads, device=cuda, generator=g).half()
        lists = ops.topk_indices(scores, nnz, torch.int32), ops.topk_indices_open_step(scores, nnz, sides[1][4], S)
        for (q, ring, k, v, state), heads, entry in zip(sides, lists, ("", "_opened")):
            _lib.call("djv_attn_step_project_batch" + entry, q.data_ptr(), w.data_ptr(), bias.data_ptr(), x.data_ptr(), ring.data_ptr(),
                      k.data_ptr(), v.data_ptr(), state.data_ptr(), heads.data_ptr(), nnz, d, nheads, hd, S, B, ops._stream())
        for a, b in zip(*sides):
            assert torch.equal(a, b), t
        assert torch.equal(sides[1][1][:, t % 16], x)


@pytest.mark.parametrize("B", [4, 5, 8, 9, 15, 16])
@pytest.mark.parametrize("nheads,hd,d,nnz", [(4, 32, 128, 4), (7, 64, 384, 5), (32, 128, 4096, 12), (40, 128, 256, 33), (6, 32, 128, 0)])
def test_output_projection_of_a_batch(cuda, B, nheads, hd, d, nnz):
    from dejavu_b200 import ops

    g = torch.Generator(device=cuda).manual_seed(B + d)
    w = (torch.randn(d, nheads, hd, device=cuda, generator=g) * max(1, nnz * hd) ** -0.5).half()
    bias, x = torch.randn(d, device=cuda, generator=g).half(), torch.randn(B, nheads, hd, device=cuda, generator=g).half()
    heads = torch.randperm(nheads, device=cuda, generator=g)[:nnz]
    want = torch.einsum("bhj,nhj->bn", x[:, heads].double(), w[:, heads].double()) + bias.double()
    near(ops.out_proj_sparse(x, w, heads.int(), bias), want)


# splits given up for blocks that fit at once: one pass and several per block, parts without tokens
@pytest.mark.parametrize("B,nheads,hd,S,length", [(16, 32, 64, 300, 290), (4, 40, 128, 700, 513), (300, 4, 32, 200, 199), (3, 32, 128, 1100, 1), (1, 72, 128, 2100, 2099)])
def test_attention_of_a_batch(cuda, B, nheads, hd, S, length):
    from dejavu_b200 import ops

    g = torch.Generator(device=cuda).manual_seed(B + S)
    q, k, v = (torch.randn(B, nheads, n, hd, device=cuda, generator=g).half() for n in (1, S, S))
    got = ops.decode_attention(q[:, :, 0], k.view(B, nheads, S, hd // 8, 8).transpose(2, 3).contiguous(), v, None, length, hd ** -0.5)
    p = (q.double() @ k[:, :, :length].double().transpose(2, 3) * hd ** -0.5).softmax(-1)
    # weights by __expf of fp32 scores: 2^-21 each beside the rounding of the result
    err = (got.double() - (p @ v[:, :, :length].double())[:, :, 0]).abs().max().item()
    assert err <= 2 ** -11 * 4 + 1e-5, err


# An error of e of a result's size takes about e / 2^-12 of the results across the edge between two fp16 values. fp32 sums are off
# by 1e-7 to 2e-7 here; sums left in the tensor cores' accumulators by 2e-6 (the projection) and 8e-7 (the output projection).
def crossed(got, want):
    return (got != want.half()).double().mean().item() * 2 ** -12


def test_sums_of_the_projections_are_those_of_fp32(cuda):
    from dejavu_b200 import _lib, ops

    g = torch.Generator(device=cuda).manual_seed(1)
    B, nheads, hd, d, S = 8, 12, 128, 9216, 16
    f16 = {"dtype": torch.float16, "device": cuda}
    w, x = (torch.randn(3, nheads, hd, d, device=cuda, generator=g) * d ** -0.5).half(), torch.randn(B, d, device=cuda, generator=g).half()
    ring, q = torch.zeros(B, 16, d, **f16), torch.zeros(B, nheads, hd, **f16)
    k, v = torch.zeros(B, nheads, hd // 8, S, 8, **f16), torch.zeros(B, nheads, S, hd, **f16)
    state = torch.zeros(_lib.ATTN_STATE_HDR + 3 * nheads, dtype=torch.int32, device=cuda)
    _lib.call("djv_attn_state_reset", state.data_ptr(), nheads, 0, ops._stream())
    _lib.call("djv_attn_step_project_batch", q.data_ptr(), w.data_ptr(), None, x.data_ptr(), ring.data_ptr(), k.data_ptr(),
              v.data_ptr(), state.data_ptr(), None, 0, d, nheads, hd, S, B, ops._stream())
    want = torch.einsum("bd,chjd->cbhj", x.double(), w.double())
    assert crossed(q, want[0]) <= 6e-7 and crossed(v[:, :, 0], want[2]) <= 6e-7
    nheads, d = 32, 4096
    w = (torch.randn(d, nheads, hd, device=cuda, generator=g) * d ** -0.5).half()
    x, heads = torch.randn(16, nheads, hd, device=cuda, generator=g).half(), torch.arange(nheads, dtype=torch.int32, device=cuda)
    assert crossed(ops.out_proj_sparse(x, w, heads), torch.einsum("bhj,nhj->bn", x.double(), w.double())) <= 5e-7
