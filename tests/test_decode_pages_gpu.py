"""Attention of single tokens over pages of any size, and its captured form."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _reference(q, k, v, lens):
    """q [B, H, D], k and v [B, G, S, D], the first lens[b] rows of each, in float64."""
    rep = q.shape[1] // k.shape[1]
    rows = []
    for b, n in enumerate(lens):
        kb, vb = (x[b, :, :n].double().repeat_interleave(rep, 0) for x in (k, v))
        s = torch.einsum("hd,hnd->hn", q[b].double(), kb) * q.shape[2] ** -0.5
        rows.append(torch.einsum("hn,hnd->hd", s.softmax(-1), vb))
    return torch.stack(rows)


# pages that hold whole key tiles (32 keys at head size 64, 16 at 128) and pages that do not; one query head per key head (multiply-add
# kernel) and groups of four (tensor cores); lengths around the ends of pages and tiles
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("page", [8, 16, 24, 32, 40])
@pytest.mark.parametrize("group", [1, 4])
def test_pages_of_any_size_match_float64(D, page, group):
    from neuronx_distributed_llama3_2_b200.ops.attention import decode_attention

    g = torch.Generator(device="cuda").manual_seed(D + page)
    lens = [1, page - 1, page, page + 1, 31, 33, 65, 8 * page, 8 * page + 17, 480]
    B, G, S = len(lens), 2, 480
    q = torch.randn(B, G * group, D, generator=g, device="cuda").bfloat16()
    k, v = (torch.randn(B, G, S, D, generator=g, device="cuda").bfloat16() for _ in range(2))
    table = torch.randperm(B * S // page, generator=g, device="cuda").reshape(B, -1)
    caches = []
    for x in (k, v):
        x = x.clone()
        for b, n in enumerate(lens):
            x[b, :, n:] = float("nan")                   # what lies behind a length is never looked at
        pages = torch.empty(B * S // page, G, page, D, dtype=x.dtype, device="cuda")
        pages[table.reshape(-1)] = x.reshape(B, G, -1, page, D).transpose(1, 2).reshape(-1, G, page, D)
        caches.append(pages)
    out = decode_attention(q, *caches, torch.tensor(lens, device="cuda"), block_table=table.to(torch.int32), page_size=page)
    ref = _reference(q, k, v, lens)
    # the weights and the result are rounded to bf16, at most 2^-8 of a value each
    assert (out.double() - ref).norm() <= 2 * 2.0 ** -8 * ref.norm()


def test_captured_steps_of_different_sizes_keep_their_scratch():
    from neuronx_distributed_llama3_2_b200.ops.attention import decode_attention

    g = torch.Generator(device="cuda").manual_seed(0)
    steps = []
    for B, S in ((2, 2048), (12, 768), (1, 4096)):       # each with partial results of another size
        q, k, v = (torch.randn(*s, generator=g, device="cuda").bfloat16() for s in ((B, 8, 128), (B, 2, S, 128), (B, 2, S, 128)))
        lens = torch.full((B,), S - 3, device="cuda")
        decode_attention(q, k, v, lens)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = decode_attention(q, k, v, lens)
        steps.append((graph, q, k, v, lens, out))
    for _ in range(2):
        for graph, q, k, v, lens, out in steps:
            q.copy_(torch.randn(q.shape, generator=g, device="cuda"))
            torch.full((1 << 22,), float("nan"), device="cuda")       # memory that a freed scratch buffer would share
            graph.replay()
            assert torch.equal(out, decode_attention(q, k, v, lens))


# one query head per key head (multiply-add kernel) and four (tensor cores)
@pytest.mark.parametrize("n_q", [2, 8])
def test_lengths_of_64_bits_are_read_as_they_are(n_q):
    from neuronx_distributed_llama3_2_b200.ops.attention import decode_attention

    g = torch.Generator(device="cuda").manual_seed(n_q)
    q = torch.randn(5, n_q, 64, generator=g, device="cuda").bfloat16()
    k, v = (torch.randn(5, 2, 640, 64, generator=g, device="cuda").bfloat16() for _ in range(2))
    lens = torch.tensor([1, 640, 129, 17, 128], device="cuda")
    ref = decode_attention(q, k, v, lens.int())
    assert torch.equal(decode_attention(q, k, v, lens), ref)
    assert torch.equal(decode_attention(q, k, v, lens.repeat_interleave(2)[::2]), ref)      # not contiguous: converted


# as many pairs of a sequence and a key head as make one split (its kernel finishes alone) and one fewer than make two, empty sequences among
# them; multiply-add kernel and tensor cores
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("group", [1, 4])
@pytest.mark.parametrize("pairs", [148, 149, 296, 297])
def test_one_split_finishes_alone(D, group, pairs):
    from neuronx_distributed_llama3_2_b200.ops.attention import decode_attention

    g = torch.Generator(device="cuda").manual_seed(pairs + D)
    q = torch.randn(pairs, group, D, generator=g, device="cuda").bfloat16()
    k, v = (torch.randn(pairs, 1, 160, D, generator=g, device="cuda").bfloat16() for _ in range(2))
    lens = torch.randint(1, 161, (pairs,), generator=g, device="cuda")
    lens[:3] = torch.tensor([160, 0, 129])
    out = decode_attention(q, k, v, lens)
    assert not out[1].any()
    real = lens > 0
    ref = _reference(q[real], k[real], v[real], lens[real].tolist())
    assert (out[real].double() - ref).norm() <= 2 * 2.0 ** -8 * ref.norm()          # as above
