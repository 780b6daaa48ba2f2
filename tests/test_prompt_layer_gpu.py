"""The prompt layer on direct kernel calls: its two kernels, and the layer against the general path."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# rows around the 256-row tile, columns around the 64-column staging and both tile widths, ragged K
@pytest.mark.parametrize("M,K,I", [(1, 8, 8), (129, 72, 40), (257, 200, 136), (300, 1024, 264), (1500, 512, 2048)])
def test_gate_up_product_with_activation_matches_float64(M, K, I):
    from neuronx_distributed_llama3_2_b200.ops.gemm import gemm_swiglu

    g = torch.Generator(device="cuda").manual_seed(M)
    wide = torch.randn(M, K + 8, generator=g, device="cuda").bfloat16()
    x, w = wide[:, :K], (torch.randn(2 * I, K, generator=g, device="cuda") * K ** -0.5 * 2).bfloat16()
    gate, up = (x.double() @ w.double().t()).chunk(2, dim=-1)
    ref = torch.nn.functional.silu(gate) * up
    # one rounding to 8 significant bits (half a unit: up to 2^-8 of a value) of fp32 sums
    assert (gemm_swiglu(x, w).double() - ref).norm() <= 2.0 ** -8 * ref.norm()


def test_gate_up_product_passes_values_that_are_no_numbers():
    from neuronx_distributed_llama3_2_b200.ops import activation
    from neuronx_distributed_llama3_2_b200.ops.gemm import gemm, gemm_swiglu

    g = torch.Generator(device="cuda").manual_seed(0)
    x, w = (torch.randn(n, 64, generator=g, device="cuda").bfloat16() for n in (300, 144))
    x[5, 3] = w[7, 0] = w[72 + 9, 1] = float("nan")                   # a row, a gate column, an up column
    w[11, 2] = w[72 + 13, 2] = float("inf")                           # infinities of both signs
    out, ref = gemm_swiglu(x, w), activation.swiglu(gemm(x, w, "nt"))
    assert ref[:, 7].isnan().all() and ref[:, 9].isnan().all() and ref.isinf().any()
    for same in (torch.isnan, torch.isposinf, torch.isneginf):
        assert torch.equal(same(out), same(ref))


@pytest.mark.parametrize("D,nq,nkv", [(16, 3, 1), (64, 8, 2), (128, 2, 2)])
@pytest.mark.parametrize("paged", [False, True])
def test_rotation_and_cache_write_match_the_separate_kernels(D, nq, nkv, paged):
    from neuronx_distributed_llama3_2_b200.ops import attention, rope

    B, T, lines, S, page = 3, 37, 5, 96, 32
    g = torch.Generator(device="cuda").manual_seed(D)
    qkv = torch.randn(B, T, nq + 2 * nkv, D, generator=g, device="cuda").bfloat16()
    cos, sin = rope.build_rope_cache(S, D, 10000.0, None, device="cuda")
    pos = torch.tensor([[0], [5], [40]], device="cuda") + torch.arange(T, device="cuda")
    sid = torch.tensor([4, 0, 2], dtype=torch.int32, device="cuda")
    shape = (lines * S // page, nkv, page, D) if paged else (lines, nkv, S, D)
    caches = [torch.zeros(shape, dtype=torch.bfloat16, device="cuda") for _ in range(4)]
    kw = {}
    if paged:
        table = torch.randperm(lines * S // page, generator=g, device="cuda").to(torch.int32).reshape(lines, -1)
        kw = {"block_table": table, "page_size": page}
    ref = rope.rope_inplace_(qkv.reshape(B * T, -1, D).clone(), cos, sin, nq + nkv, positions=pos.reshape(-1)).view(qkv.shape)
    attention.kv_cache_update(caches[0], caches[1], ref[:, :, nq:nq + nkv].permute(0, 2, 1, 3),
                              ref[:, :, nq + nkv:].permute(0, 2, 1, 3), pos[:, 0], seq_ids=sid, **kw)
    out = rope.rope_cache_write_(qkv.clone(), cos, sin, pos.to(torch.int32).contiguous(), caches[2], caches[3], nq, nkv, seq_ids=sid,
                                 **kw)
    for a, b in ((out, ref), (caches[2], caches[0]), (caches[3], caches[1])):
        # the same two products and a sum in fp32: fused or not, one unit in the last place of bf16
        assert torch.equal(a == 0, b == 0) and ((a - b).abs().float() <= 2.0 ** -7 * b.abs().float()).all()


@pytest.mark.parametrize("D,B,T,paged", [(64, 1, 200, False), (128, 3, 77, True)])
def test_prompt_layer_matches_the_general_path(D, B, T, paged, monkeypatch):
    from neuronx_distributed_llama3_2_b200.inference.config import InferenceConfig
    from neuronx_distributed_llama3_2_b200.inference.model import KVCacheInferenceMixin, LlamaInferenceModel
    from neuronx_distributed_llama3_2_b200.models.llama import LlamaConfig

    torch.manual_seed(0)
    cfg = LlamaConfig(vocab_size=512, hidden_size=256, intermediate_size=520, num_hidden_layers=2, num_attention_heads=4,
                      num_key_value_heads=2, head_dim=D, rope_scaling=None, initializer_range=0.05)
    model = LlamaInferenceModel(cfg, InferenceConfig(batch_size=B, max_batch_size=4, max_context_length=256, seq_len=256,
                                                     is_continuous_batching=True, paged_kv=paged, page_size=64), device="cuda")
    ids = torch.randint(0, 512, (B, T), device="cuda")
    pos = torch.arange(T, device="cuda").expand(B, T)
    lines, last = torch.tensor([2, 0, 3], dtype=torch.int32, device="cuda")[:B], torch.tensor([T - 1, 3, 50], device="cuda")[:B]
    taken = []
    real = KVCacheInferenceMixin._layer_prompt
    monkeypatch.setattr(KVCacheInferenceMixin, "_layer_prompt", lambda self, *a: taken.append(1) or real(self, *a))

    def run():
        cache = model.init_kv_cache(device="cuda")
        logits = model.forward_infer(ids, pos, lines, last, return_logits=True, sample=False)[1]
        return logits, cache.k + cache.v

    got, got_cache = run()
    assert len(taken) == 2
    hook = model.model.layers[0].mlp.register_forward_hook(lambda *a: None)      # a hooked layer keeps the general path
    run()
    assert len(taken) == 3
    hook.remove()
    monkeypatch.setattr(KVCacheInferenceMixin, "_prompt_layer_ok", lambda *a: False)
    ref, ref_cache = run()
    # the general path rounds gate and up to bf16 ahead of the activation (2^-9 each); two layers of such differences
    for a, b in zip([got] + got_cache, [ref] + ref_cache):
        assert (a.float() - b.float()).norm() <= 2e-2 * b.float().norm()


def test_hooks_on_every_module_see_the_prompt_layer(monkeypatch):
    from neuronx_distributed_llama3_2_b200.inference.config import InferenceConfig
    from neuronx_distributed_llama3_2_b200.inference.model import KVCacheInferenceMixin, LlamaInferenceModel
    from neuronx_distributed_llama3_2_b200.models.llama import LlamaConfig

    cfg = LlamaConfig(vocab_size=512, hidden_size=256, intermediate_size=512, num_hidden_layers=1, num_attention_heads=4,
                      num_key_value_heads=2, head_dim=64, rope_scaling=None)
    model = LlamaInferenceModel(cfg, InferenceConfig(batch_size=1, max_context_length=256, seq_len=256), device="cuda")
    model.init_kv_cache(device="cuda")
    ids, pos = torch.randint(0, 512, (1, 200), device="cuda"), torch.arange(200, device="cuda").unsqueeze(0)

    def seen(register):
        names, handle = [], register(lambda m, *a: names.append(type(m).__name__))
        try:
            model.forward_infer(ids, pos, sample=False)
        finally:
            handle.remove()
        return names

    every = torch.nn.modules.module
    registers = (every.register_module_forward_hook, every.register_module_forward_pre_hook)
    names = [seen(r) for r in registers]
    monkeypatch.setattr(KVCacheInferenceMixin, "_prompt_layer_ok", lambda *a: False)
    assert names == [seen(r) for r in registers] and "GQAQKVColumnParallelLinear" in names[0]
