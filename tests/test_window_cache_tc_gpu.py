"""Attention of a portion of tokens over the KV cache on the tcgen05 kernel, against the fp32 restatement."""
import pytest
import torch

pytestmark = pytest.mark.gpu

FORMS = ["plain", "window", "kept", "sinks", "capped", "sigmoid", "gated", "columns"]


@pytest.mark.parametrize("D", [64, 128])
# portions around the 128-row query tile, starts around the 64-row key tile, padded and empty rows
@pytest.mark.parametrize("T,starts,n_new", [(64, [0, 1, 63], None), (65, [64, 700, 129], [65, 1, 0]), (200, [5, 0, 333], [129, 200, 64]),
                                            (300, [128, 20, 961], None)])
@pytest.mark.parametrize("page", [0, 64, 128])
@pytest.mark.parametrize("form", FORMS)
def test_portion_over_the_cache_matches_the_restatement(D, T, starts, n_new, page, form):
    from neuronx_distributed_llama3_2_b200.ops import window_attention as wa

    B, H, G, lines = len(starts), 4, 2, 5
    g = torch.Generator(device="cuda").manual_seed(T + D + page)

    def normal(*s):
        return torch.randn(*s, generator=g, device="cuda")

    S = 1408                                            # rows of a line, a multiple of the pages
    line = torch.tensor([3, 0, 2], dtype=torch.int32, device="cuda")
    k, v = (normal(lines, G, S, D).bfloat16() for _ in range(2))
    ends = [s + (T if n_new is None else n) for s, n in zip(starts, n_new or starts)]
    for b, e in enumerate(ends):                        # what lies behind a sequence's end is never looked at
        k[line[b], :, e:] = float("nan")
        v[line[b], :, e:] = float("nan")
    q = normal(B, T, H, D).bfloat16()
    kw = {"window": {}, "plain": {}, "kept": {"keep_first": 70}, "sinks": {"sinks": normal(H)},
          "capped": {"softcap": 3.0, "log_bias": (normal(H).abs(), normal(H).abs())},
          "sigmoid": {"sigmoid_bias": normal(H), "softcap": 20.0}, "gated": {"gate": normal(B, T, H).bfloat16()},
          "columns": {"gate": normal(B, T, H * D).bfloat16(), "gate_elements": True, "gate_mul": 2.0}}[form]
    window = None if form in ("plain", "sinks") else 100
    slopes = wa.distance_slopes(H, device="cuda") if form in ("window", "kept", "gated") else None
    new = None if n_new is None else torch.tensor(n_new, dtype=torch.int32, device="cuda")
    start = torch.tensor(starts, dtype=torch.int32, device="cuda")
    ck, cv, paged = k, v, {}
    if page:
        table = torch.randperm(lines * S // page, generator=g, device="cuda").reshape(lines, -1)
        ck, cv = torch.empty(lines * S // page, G, page, D, dtype=k.dtype, device="cuda"), None
        cv = torch.empty_like(ck)
        for dst, src in ((ck, k), (cv, v)):
            dst[table.reshape(-1)] = src.reshape(lines, G, -1, page, D).transpose(1, 2).reshape(-1, G, page, D)
        paged = {"block_table": table.to(torch.int32), "page_size": page}
    wide = torch.full((B * T, H * D + 64), 7.0, dtype=q.dtype, device="cuda")
    out = wa.window_attention_prefill(q, ck, cv, start, D ** -0.5, window, slopes=slopes, n_new=new, seq_ids=line, impl="tc",
                                      out=wide[:, 32:32 + H * D], **kw, **paged).reshape(B, T, H, D)
    assert (wide[:, :32] == 7).all() and (wide[:, -32:] == 7).all()
    gate = kw.pop("gate", None)
    keep = kw.pop("keep_first", 0)
    for b in range(B):
        n, e = ends[b] - starts[b], ends[b]
        assert not out[b, n:].any()                     # padding rows come out as zeros
        if n == 0:
            continue
        ref = wa.window_attention_ref(q[b, :n], k[line[b], :, :e], v[line[b], :, :e], torch.arange(starts[b], e, device="cuda"),
                                      D ** -0.5, window, keep, slopes, gate=None if gate is None else gate[b, :n], **kw)
        # the weights and the result are rounded to bf16: 2^-9 of each weight and of the value
        assert (out[b, :n].float() - ref).norm() <= 2.0 ** -7 * ref.norm()


# weights are rounded to bf16: relative to the row's running maximum the largest one is 1 and keeps its value, relative to a stale
# maximum it is rounded too.  Few keys that matter (distance bias, scores of a wide spread), and many
@pytest.mark.parametrize("D,T,past,window,bias,spread", [(128, 300, 600, 512, True, 1.0), (64, 300, 100, None, False, 1.0),
                                                         (64, 300, 600, 512, False, 3.0), (128, 200, 3000, None, True, 2.0)])
def test_weights_are_no_further_off_than_on_the_mma_kernel(D, T, past, window, bias, spread):
    from neuronx_distributed_llama3_2_b200.ops import window_attention as wa

    B, H, G, S = 2, 16, 4, past + T
    g = torch.Generator(device="cuda").manual_seed(D + T)
    q, k, v = (torch.randn(*s, generator=g, device="cuda").bfloat16() for s in ((B, T, H, D), (B, G, S, D), (B, G, S, D)))
    q = q * spread
    slopes = wa.distance_slopes(H, device="cuda") if bias else None
    start = torch.full((B,), past, dtype=torch.int32, device="cuda")
    pos, key = torch.arange(past, S, device="cuda"), torch.arange(S, device="cuda")
    dist = pos[:, None] - key[None]
    s = torch.einsum("bthd,bhnd->bhtn", q.double(), k.double().repeat_interleave(H // G, 1)) * D ** -0.5
    if bias:
        s -= slopes.double()[:, None, None] * dist
    s.masked_fill_((dist < 0) | (dist >= (window or S)), float("-inf"))
    ref = torch.einsum("bhtn,bhnd->bthd", s.softmax(-1), v.double().repeat_interleave(H // G, 1))
    tc, mma = ((wa.window_attention_prefill(q, k, v, start, D ** -0.5, window, slopes=slopes, impl=i).double() - ref).norm()
               for i in ("tc", "mma"))
    # both errors are sums over more than 6000 rows of independent roundings, their ratio scatters by less than 2 %
    assert tc <= 1.02 * mma


# on either side of the 16 tokens from which weights are rounded to bf16, over a cache that is long enough for any portion
@pytest.mark.parametrize("T,kernel", [(2, "generic"), (15, "generic"), (16, "tc")])
def test_few_tokens_over_a_long_cache_keep_fp32_weights(T, kernel):
    from neuronx_distributed_llama3_2_b200.ops import window_attention as wa

    g = torch.Generator(device="cuda").manual_seed(T)
    q, k, v = (torch.randn(*s, generator=g, device="cuda").bfloat16() for s in ((1, T, 4, 128), (1, 2, 1 << 17, 128), (1, 2, 1 << 17, 128)))
    start = torch.full((1,), 500, dtype=torch.int32, device="cuda")
    assert T * k.shape[2] >= wa.TC_CACHE_MIN_WORK
    auto, same = (wa.window_attention_prefill(q, k, v, start, 0.1, 300, impl=i) for i in ("auto", kernel))
    assert torch.equal(auto, same)


# windows and kept first rows around the 64-row key tile; the oldest visible key scores highest, so that the running maximum moves in
# every tile on the way back from the diagonal, and the first tiles of a row may hold nothing that it sees
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("window,keep", [(1, 0), (63, 1), (64, 64), (65, 63), (64, 65), (129, 130), (500, 3)])
def test_masks_and_the_order_of_the_tiles(D, window, keep):
    from neuronx_distributed_llama3_2_b200.ops import window_attention as wa

    B, T, H, G = 2, 200, 4, 2
    g = torch.Generator(device="cuda").manual_seed(D + window)
    starts, S = [333, 5], 640
    q = torch.ones(B, T, H, D, device="cuda") + 0.1 * torch.randn(B, T, H, D, generator=g, device="cuda")
    k = torch.linspace(2, -2, S, device="cuda")[:, None] + 0.1 * torch.randn(B, G, S, D, generator=g, device="cuda")
    q, k, v = q.bfloat16(), k.bfloat16(), torch.randn(B, G, S, D, generator=g, device="cuda").bfloat16()
    out = wa.window_attention_prefill(q, k, v, torch.tensor(starts, dtype=torch.int32, device="cuda"), D ** -0.5, window, keep, impl="tc")
    for b, s in enumerate(starts):
        ref = wa.window_attention_ref(q[b], k[b, :, :s + T], v[b, :, :s + T], torch.arange(s, s + T, device="cuda"), D ** -0.5, window, keep,
                                      None)
        assert (out[b].float() - ref).norm() <= 2.0 ** -7 * ref.norm()          # weights and result in bf16, as above
