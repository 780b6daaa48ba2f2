"""Token steps of 1 to 8 rows on the tensor-core weight-streaming kernels, against float64 and the FMA kernels."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 2, 5, 8])
# around the line between the kernels, ragged last weight slabs and contraction tails
@pytest.mark.parametrize("n,k", [(1024, 2048), (2056, 1032), (264, 1024), (16, 8192), (2056, 4104)])
def test_few_rows_match_float64(rows, n, k):
    from neuronx_distributed_llama3_2_b200.ops.linear import gemm_nt

    g = torch.Generator(device="cuda").manual_seed(n + rows)
    x, w = (torch.randn(r, k, generator=g, device="cuda").bfloat16() for r in (rows, n))
    ref = x.double() @ w.double().t()
    # one rounding to 8 significant bits (half a unit: up to 2^-8 of a value) of an fp32 sum
    assert (gemm_nt(x, w).double() - ref).norm() <= 2.0 ** -8 * ref.norm()


# one CTA per SM: 12 weight slabs in clusters of 8, 13 in clusters of 4
@pytest.mark.parametrize("n", [1536, 1544])
def test_many_rows_match_float64(n):
    test_few_rows_match_float64(100, n, 2048)


@pytest.mark.parametrize("batch,paged", [(2, False), (3, True), (8, False)])
def test_token_step_matches_the_fma_kernels(batch, paged, monkeypatch):
    from neuronx_distributed_llama3_2_b200.inference.config import InferenceConfig
    from neuronx_distributed_llama3_2_b200.inference.model import KVCacheInferenceMixin, LlamaInferenceModel
    from neuronx_distributed_llama3_2_b200.models.llama import LlamaConfig

    torch.manual_seed(0)
    cfg = LlamaConfig(vocab_size=512, hidden_size=1536, intermediate_size=2048, num_hidden_layers=2, num_attention_heads=12,
                      num_key_value_heads=4, head_dim=128, rope_scaling=None)
    model = LlamaInferenceModel(cfg, InferenceConfig(batch_size=batch, max_context_length=64, seq_len=64, paged_kv=paged,
                                                     page_size=32), device="cuda")
    ids = torch.randint(0, 512, (batch, 1), device="cuda")
    pos = torch.arange(5, 5 + batch, device="cuda").reshape(batch, 1)
    taken = []
    real = KVCacheInferenceMixin._layer_batched_decode
    monkeypatch.setattr(KVCacheInferenceMixin, "_layer_batched_decode", lambda self, *a: taken.append(1) or real(self, *a))

    def run():
        cache = model.init_kv_cache(device="cuda")
        g = torch.Generator(device="cuda").manual_seed(1)
        for t in cache.k + cache.v:
            t.normal_(generator=g)
        logits = model.forward_infer(ids, pos, return_logits=True, sample=False)[1]
        return [logits] + cache.k + cache.v

    got = run()
    assert len(taken) == 2
    monkeypatch.setattr(KVCacheInferenceMixin, "_tensor_core_decode", lambda *a: False)
    ref = run()
    assert len(taken) == 2
    for a, b in zip(got, ref):      # the same roundings to bf16 of fp32 sums in another order, two layers of them
        assert (a.float() - b.float()).norm() <= 1e-2 * b.float().norm()


@pytest.mark.parametrize("paged", [False, True])
def test_one_sequence_matches_the_fma_kernels(paged, monkeypatch):
    test_token_step_matches_the_fma_kernels(1, paged, monkeypatch)


@pytest.mark.parametrize("rows", [1, 2, 3, 4])
# widths whose last block of 64 columns is not full, a contraction that is split unevenly, heads of both sizes
@pytest.mark.parametrize("K,n_q,n_kv,D,I", [(2048, 32, 8, 64, 8192), (1032, 4, 4, 128, 264), (520, 24, 8, 128, 4096)])
def test_norm_inside_the_projections(rows, K, n_q, n_kv, D, I):
    from neuronx_distributed_llama3_2_b200.ops import decode_fused as df, norm, rope

    g = torch.Generator(device="cuda").manual_seed(K + rows)
    x = (torch.randn(rows, 2 * K, generator=g, device="cuda").bfloat16() * 3)[:, :K]        # a row pitch of its own
    assert x.stride(0) == 2 * K
    nw = (torch.randn(K, generator=g, device="cuda") * 0.1 + 1).bfloat16()
    w_qkv = torch.randn((n_q + 2 * n_kv) * D, K, generator=g, device="cuda").bfloat16() * 0.02
    w_gu = torch.randn(2 * I, K, generator=g, device="cuda").bfloat16() * 0.02
    cos, sin = rope.build_rope_cache(64, D, 1e4, None, device="cuda")
    pos = torch.arange(3, 3 + rows, device="cuda").int()
    assert df.norm_fits(x, w_qkv, False) and df.norm_fits(x, w_gu, True)
    assert not df.norm_fits(torch.empty(5, K, dtype=torch.bfloat16, device="cuda"), w_qkv, False)
    caches = [torch.zeros(4, rows, n_kv, 32, D, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    xn = norm.rms_norm(x.contiguous(), nw, 1e-5)
    got = [df.norm_qkv_rope_cache(x, nw, 1e-5, w_qkv, cos, sin, pos, caches[0][0], caches[0][1], n_q, n_kv, D), caches[0],
           df.norm_gate_up_swiglu(x, nw, 1e-5, w_gu)]
    ref = [df.qkv_rope_cache_batched(xn, w_qkv, cos, sin, pos, caches[1][0], caches[1][1], n_q, n_kv, D), caches[1],
           df.gate_up_swiglu_batched(xn, w_gu)]
    # the same roundings; only the sum of squares is in another order, which moves some activations to the neighbouring bf16 value
    for a, b in zip(got, ref):
        assert (a.float() - b.float()).norm() <= 1e-3 * b.float().norm()
