"""The sparse mixture on rows that are sorted by expert on the device, and the router, against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _reference(h, idx, wts, w_in, w_down, limit, alpha, shift, scale_input):
    h, w_in, w_down = h.double(), w_in.double(), w_down.double()
    E, y = w_in.shape[0], torch.zeros_like(h)
    for j in range(idx.shape[1]):
        for e in range(E):
            rows = (idx[:, j] == e).nonzero()[:, 0]
            w = wts[rows, j].double().unsqueeze(1)
            z = ((h[rows] * w) if scale_input else h[rows]) @ w_in[e]
            if limit is None:
                a = z.clamp(min=0).square()
            else:
                g, u = z.chunk(2, dim=-1)
                g, u = g.clamp(max=limit), u.clamp(-limit, limit)
                a = g * torch.sigmoid(alpha * g) * (u + shift)
            y[rows] += (a @ w_down[e]) * (1.0 if scale_input else w)
        rows = (idx[:, j] >= E).nonzero()[:, 0]
        y[rows] += wts[rows, j].double().unsqueeze(1) * h[rows]
    return y


# tokens around the 32-row alignment, the 128- / 256-row tiles and empty experts; widths around the 64-column staging and the
# 128 / 256-column tiles; the most experts
@pytest.mark.parametrize("N,E,top,W,F", [(1, 3, 2, 8, 8), (31, 1, 1, 72, 40), (33, 5, 2, 136, 72), (257, 4, 4, 264, 200),
                                         (1000, 7, 3, 64, 136), (700, 128, 2, 128, 64), (3000, 2, 1, 1024, 512)])
@pytest.mark.parametrize("form", ["glu", "input", "relu2"])
def test_sorted_experts_match_float64(N, E, top, W, F, form):
    from neuronx_distributed_llama3_2_b200.ops import moe_sparse as ms

    g = torch.Generator(device="cuda").manual_seed(N + E)

    def normal(*s):
        return torch.randn(*s, generator=g, device="cuda")

    h = normal(N, W).bfloat16()
    w_in = (normal(E, W, F if form == "relu2" else 2 * F) * W ** -0.5).bfloat16()
    w_down = (normal(E, F, W) * F ** -0.5).bfloat16()
    # expert 0 is never chosen when there is another one; index E is an identity expert
    idx = torch.randint(min(1, E - 1), E + 1, (N, top), generator=g, device="cuda").to(torch.int32)
    wts = torch.rand(N, top, generator=g, device="cuda") + 0.1
    scale_input = form == "input"
    limit = None if form == "relu2" else 1.5
    Fs = F + 8
    s_in, s_down = (normal(1, W, Fs if form == "relu2" else 2 * Fs) * W ** -0.5).bfloat16(), (normal(1, Fs, W) * Fs ** -0.5).bfloat16()
    gate = torch.rand(N, generator=g, device="cuda")
    assert ms.sorted_forward_applies(h, w_in, w_down, s_in, s_down)
    ones = torch.where(idx < E, torch.ones_like(wts), wts)
    out = ms.sorted_forward(h, idx, ones if scale_input else wts, w_in, w_down, limit is not None, limit or 0.0, 1.7, 1.0,
                            wts if scale_input else None, s_in, s_down, 0.8, gate)
    ref = _reference(h, idx, wts, w_in, w_down, limit, 1.7, 1.0, scale_input)
    every = torch.zeros(N, 1, dtype=torch.int32, device="cuda")
    ref += _reference(h, every, gate.unsqueeze(1), s_in, s_down, None if limit is None else 0.8, 1.7, 1.0, False)
    # the activation is rounded to bf16, at most 2^-8 of a value; the errors of different terms are independent, so their sum stays
    # below that share of the sum; fp32 sums
    assert (out.double() - ref).norm() <= 2.0 ** -8 * ref.norm()


@pytest.mark.parametrize("N,W,R", [(5, 72, 3), (5, 50, 37), (2400, 64, 37), (2401, 50, 9), (2369, 200, 700)]
                         # a CTA, a warp and a quarter of a warp per token, the last with vector and with scalar loads
                         + [(1183, 72, 5), (1185, 72, 5), (3601, 256, 40), (9601, 50, 80)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_router_forms_match_float64(N, W, R, dtype):
    from neuronx_distributed_llama3_2_b200.ops import moe_sparse as ms

    g = torch.Generator(device="cuda").manual_seed(N)
    h = torch.randn(N, W, generator=g, device="cuda").to(dtype)
    w = torch.randn(R, W, generator=g, device="cuda") * W ** -0.5
    gate = torch.randn(1, W, generator=g, device="cuda") * W ** -0.5
    idx, wts, sg = ms.route(h, w, None, 2, 1.5, gate)
    z = h.double() @ w.double().t()
    p = torch.softmax(z, dim=-1)
    top = torch.topk(p, 2, dim=-1)
    # fp32 sums of W terms: a choice may differ only between scores that are closer than their rounding
    assert (p.gather(1, idx.long()) - top.values).abs().max() <= 1e-5
    assert (wts.double() - 1.5 * p.gather(1, idx.long())).abs().max() <= 1e-5
    assert (sg.double() - torch.sigmoid(h.double() @ gate.double()[0])).abs().max() <= 1e-5


# a token's CTA splits the width between its warps: four and eight of them (3 tokens per SM), parts that do not divide the warps, widths of
# fewer pieces than parts, outputs of one to nine groups of four
@pytest.mark.parametrize("N,W,R", [(1, 4096, 8), (7, 2048, 12), (9, 2056, 1), (3, 264, 5), (2, 33, 9), (444, 520, 33), (445, 520, 8), (1183, 1000, 8)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_warps_that_share_a_token_match_float64(N, W, R, dtype):
    from neuronx_distributed_llama3_2_b200.ops import moe_sparse as ms

    g = torch.Generator(device="cuda").manual_seed(N + W)
    h = torch.randn(N, W, generator=g, device="cuda").to(dtype)
    w = torch.randn(R, W, generator=g, device="cuda") * W ** -0.5
    gate = torch.randn(1, W, generator=g, device="cuda") * W ** -0.5
    bias = torch.randn(R, generator=g, device="cuda")
    idx, wts, sg = ms.route(h, w, None, 1, 1.5, gate, logit_bias=bias)
    p = torch.softmax(h.double() @ w.double().t() + bias.double(), dim=-1)
    chosen = p.gather(1, idx.long())
    # fp32 sums of W terms of size 1: a choice may differ only between scores that are closer than their rounding
    assert (chosen[:, 0] - p.amax(-1)).abs().max() <= 1e-5
    assert (wts.double() - 1.5 * chosen).abs().max() <= 1e-5
    assert (sg.double() - torch.sigmoid(h.double() @ gate.double()[0])).abs().max() <= 1e-5

# below and above 16 pairs per expert (32 tokens), one and several row tiles; with and without a shared expert
@pytest.mark.parametrize("N", [1, 31, 32, 200, 1000])
@pytest.mark.parametrize("shared", [0, 72])
def test_captured_step_repeats_and_is_as_exact_as_the_pairs(N, shared):
    from neuronx_distributed_llama3_2_b200.modules.moe.sparse import SparseMoE

    g = torch.Generator(device="cuda").manual_seed(N + shared)
    m = SparseMoE(136, 4, 2, 200, 1.5, shared_intermediate_size=shared, dtype=torch.bfloat16, device="cuda").eval()
    with torch.no_grad():
        for p in m.parameters():
            p.copy_(torch.randn(p.shape, generator=g, device="cuda") * p.shape[-2] ** -0.5 if p.dim() > 1 else torch.zeros_like(p))
        h, first = (torch.randn(N, 136, generator=g, device="cuda").bfloat16() for _ in range(2))
        given = first.clone()
        m(given, path="device")
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = m(given, path="device")
        for x in (first, h, first, h):                  # every replay reads its own input
            given.copy_(x)
            graph.replay()
            assert torch.equal(out, m(x, path="device"))
        idx, wts, gate = m.router.select(h, m.shared_gate.weight if shared else None)
        ref = _reference(h, idx, wts, m.experts.gate_up_proj.weight, m.experts.down_proj.weight, 1.5, 1.702, 1.0, False)
        if shared:
            ref += _reference(h, torch.zeros(N, 1, dtype=torch.int32, device="cuda"), gate.unsqueeze(1),
                              m.shared.gate_up_proj.weight, m.shared.down_proj.weight, 1.5, 1.702, 1.0, False)
        ours, pairs = ((y.double() - ref).norm() for y in (out, m(h, path="pairs")))
    # both round the activation to bf16 and nothing else, at the same values but for those next to a rounding boundary (a second
    # rounding, of the experts' outputs, would make it 1.4)
    assert ours <= 1.1 * pairs


def test_each_path_is_the_one_that_was_asked_for(monkeypatch):
    from neuronx_distributed_llama3_2_b200.modules.moe.sparse import SparseMoE

    g = torch.Generator(device="cuda").manual_seed(5)
    m = SparseMoE(128, 4, 2, 64, 1.5, dtype=torch.bfloat16, device="cuda").eval()
    taken = []
    for name in ("_forward_sorted", "_forward_device_sorted"):
        monkeypatch.setattr(m, name, lambda *a, name=name, call=getattr(m, name): (taken.append(name), call(*a))[1])
    with torch.no_grad():
        for p in m.parameters():
            p.copy_(torch.randn(p.shape, generator=g, device="cuda") * 0.1)
        h = torch.randn(90, 128, generator=g, device="cuda").bfloat16()
        by_path = {path: m(h, path=path) for path in ("pairs", "sorted", "device", None)}
        assert taken == ["_forward_sorted", "_forward_device_sorted"]
        assert torch.equal(by_path["pairs"], by_path[None])                  # 90 tokens of a small mixture
        many = torch.randn(3000, 128, generator=g, device="cuda").bfloat16()
        assert torch.equal(m(many), m(many, path="device")) and taken[2:] == ["_forward_device_sorted"] * 2
    # the host-counted path rounds the experts' outputs to bf16, all round the activation: 2^-8 of a value each
    for y in by_path.values():
        assert (y - by_path["pairs"]).norm() <= 3 * 2.0 ** -8 * by_path["pairs"].norm()


# around the pairs that one launch sorts (2048), identity experts, a shared expert with its gate, every form of the scores
@pytest.mark.parametrize("tokens", [64, 511, 512, 513])
@pytest.mark.parametrize("kw", [dict(), dict(num_identity_experts=3, shared_intermediate_size=128, normalize=True),
                                dict(score="sigmoid", router_bias=True, shared_intermediate_size=64, shared_gated=False),
                                dict(renormalize=True, gated=False)])
def test_router_and_experts_in_one_call(tokens, kw):
    from neuronx_distributed_llama3_2_b200.modules.moe.sparse import SparseMoE

    torch.manual_seed(tokens)
    m = SparseMoE(512, 12, 4, 256, 7.0, dtype=torch.bfloat16, device="cuda", **kw).eval()
    with torch.no_grad():
        for p in m.parameters():
            p.normal_(0, 0.05)
        h = torch.randn(tokens, 512, device="cuda").bfloat16()
        calls, select = [], m.router.select
        whole = m(h)
        m.router.select = lambda *a: calls.append(1) or select(*a)      # a replaced router is asked
        assert torch.equal(m(h), whole) and len(calls) == 1
        assert torch.equal(m(h, path="device"), whole)
        pairs = m(h, path="pairs")
    # the per-pair kernels: bf16 activations of fp32 sums in another order
    assert (whole - pairs).norm() <= 2.0 ** -8 * pairs.norm()


@pytest.mark.parametrize("path", [None, "device", "pairs", "sorted"])
@pytest.mark.parametrize("kw", [dict(score="sigmoid", normalize=True), dict(score="sigmoid", renormalize=True)])
def test_router_forms_that_do_not_exist_are_refused_on_every_path(path, kw):
    from neuronx_distributed_llama3_2_b200.modules.moe.sparse import SparseMoE

    m = SparseMoE(512, 12, 4, 256, 7.0, dtype=torch.bfloat16, device="cuda", **kw).eval()
    with torch.no_grad(), pytest.raises(AssertionError):
        m(torch.zeros(64, 512, device="cuda").bfloat16(), path=path)
