"""The prompt pass of the sparse decoder: what goes into the caches, and which tokens get logits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,L,nheads,hd,S", [(1, 1, 3, 32, 1), (2, 31, 2, 64, 40), (1, 33, 5, 128, 33), (3, 130, 4, 32, 200), (1, 1983, 2, 128, 1999)])
def test_prompt_keys_and_values_go_to_their_places(cuda, B, L, nheads, hd, S):
    from dejavu_b200 import ops

    g = torch.Generator(device=cuda).manual_seed(L)
    qkv = torch.randn(B, L, 3, nheads, hd, device=cuda, generator=g).half()
    k = torch.randn(B, nheads, hd // 8, S, 8, device=cuda, generator=g).half()
    v = torch.randn(B, nheads, S, hd, device=cuda, generator=g).half()
    want_k, want_v = k.clone(), v.clone()
    want_k[:, :, :, :L] = qkv[:, :, 1].reshape(B, L, nheads, hd // 8, 8).permute(0, 2, 3, 1, 4)
    want_v[:, :, :L] = qkv[:, :, 2].transpose(1, 2)
    ops.kv_store(k, v, qkv)
    assert torch.equal(k, want_k) and torch.equal(v, want_v)


@pytest.mark.parametrize("B,n,rows", [(1, 7, [6]), (2, 5, [-1]), (1, 1, [0]), (3, 6, [0, 4]), (1, 4, []), (2, 3, [0, 1, 2])])
def test_logits_of_chosen_tokens(cuda, B, n, rows):
    from dejavu_b200.generation import InferenceParams, allocate_kv_cache, step
    from dejavu_b200.gpt import GPTLMHeadModel, apply_sparsity_knobs, opt_config

    cfg = apply_sparsity_knobs(opt_config("opt-125m", n_layer=2, n_embd=256, hidden_size=256, n_head=4, n_inner=1024, vocab_size=520,
                                          max_position_embeddings=64, mlp_sp_dim=64, att_sp_dim=32), 256, 2, 2)
    model = GPTLMHeadModel(cfg, device=cuda, dtype=torch.float16).eval().init_random(0, std=0.05)
    ids = torch.randint(0, 512, (B, n), generator=torch.Generator().manual_seed(n)).to(cuda)
    out = []
    for wanted in (None, rows):
        ip = InferenceParams(max_sequence_len=n, max_batch_size=B, key_value_memory_dict=allocate_kv_cache(model, B, n, cuda))
        out.append(step(model, ip, ids, logit_rows=wanted))
    assert out[1].shape == (B, len(rows), out[0].size(2))
    # two products of 256 terms in fp32, each rounded to fp16
    assert (out[1] - out[0][:, rows]).abs().le(2 ** -10 * out[0].abs().max() + 1e-5).all()


def test_the_head_of_a_prompt_is_a_module_that_is_called(cuda):
    from dejavu_b200.generation import InferenceParams, allocate_kv_cache, step
    from dejavu_b200.gpt import GPTLMHeadModel, apply_sparsity_knobs, opt_config

    cfg = apply_sparsity_knobs(opt_config("opt-125m", n_layer=2, n_embd=256, hidden_size=256, n_head=4, n_inner=1024, vocab_size=520,
                                          max_position_embeddings=64, mlp_sp_dim=64, att_sp_dim=32), 256, 2, 2)
    model = GPTLMHeadModel(cfg, device=cuda, dtype=torch.float16).eval().init_random(0, std=0.05)
    model.lm_head.register_forward_hook(lambda head, args, result: 2 * result)
    ids = torch.arange(5, device=cuda)[None]
    out = []
    for rows in (None, [4]):
        ip = InferenceParams(max_sequence_len=5, max_batch_size=1, key_value_memory_dict=allocate_kv_cache(model, 1, 5, cuda))
        out.append(step(model, ip, ids, logit_rows=rows))
    assert (out[1] - out[0][:, [4]]).abs().le(2 ** -9 * out[0].abs().max() + 1e-5).all()  # (products of 256 terms, rounded to fp16)


def test_a_prompt_without_tokens_leaves_empty_caches(cuda):
    from dejavu_b200.generation import InferenceParams, allocate_kv_cache, step
    from dejavu_b200.gpt import GPTLMHeadModel, apply_sparsity_knobs, opt_config

    cfg = apply_sparsity_knobs(opt_config("opt-125m", n_layer=2, n_embd=256, hidden_size=256, n_head=4, n_inner=1024, vocab_size=520,
                                          max_position_embeddings=64, mlp_sp_dim=64, att_sp_dim=32), 256, 2, 2)
    model = GPTLMHeadModel(cfg, device=cuda, dtype=torch.float16).eval().init_random(0, std=0.05)
    ip = InferenceParams(max_sequence_len=4, max_batch_size=1, key_value_memory_dict=allocate_kv_cache(model, 1, 4, cuda))
    assert step(model, ip, torch.zeros(1, 0, dtype=torch.long, device=cuda)).shape == (1, 0, 520)
