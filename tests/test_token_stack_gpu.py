"""All decoder layers of a one-sequence step in one launch, against the layers kernel by kernel and against float64."""
import copy

import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = {"64": (2048, 8192, 32, 8, 64), "128": (3072, 8192, 24, 8, 128)}      # hidden, feed-forward, heads, key / value heads, head size
EPS = 1e-5


def _draw(size, layers, lines, rows, seed):
    H, I, nq, nkv, D = SIZES[size]
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape, std=0.02, mean=0.0):
        return torch.empty(shape, dtype=torch.bfloat16, device="cuda").normal_(mean, std, generator=gen)

    return [[normal(H, std=0.1, mean=1.0), normal((nq + 2 * nkv) * D, H), normal(H, nq * D), normal(H, std=0.1, mean=1.0),
             normal(2 * I, H), normal(H, I), normal(lines, nkv, rows, D, std=1.0), normal(lines, nkv, rows, D, std=1.0)]
            for _ in range(layers)], normal(1, H, std=1.0)


def _tables(D, rows):
    ang = torch.outer(torch.arange(rows, dtype=torch.float64), 500000.0 ** (-torch.arange(0, D, 2, dtype=torch.float64) / D))
    return ang.cos().float().cuda(), ang.sin().float().cuda()


def _chain(x, layers, size, cos, sin, pos, lens, **place):
    from neuronx_distributed_llama3_2_b200.ops import decode_fused as df
    from neuronx_distributed_llama3_2_b200.ops.attention import decode_attention
    from neuronx_distributed_llama3_2_b200.ops.gemm import gemm_smallm
    from neuronx_distributed_llama3_2_b200.ops.norm import rms_norm

    H, I, nq, nkv, D = SIZES[size]
    for n1, wqkv, wo, n2, wgu, wd, ck, cv in layers:
        q = df.qkv_rope_cache_batched(rms_norm(x, n1, EPS), wqkv, cos, sin, pos, ck, cv, nq, nkv, D, **place)
        o = decode_attention(q, ck, cv, lens, block_table=place.get("block_table"), page_size=place.get("page_size", 0),
                             seq_ids=place.get("seq_ids")).reshape(1, nq * D)
        x = gemm_smallm(o, wo, residual=x)
        x = gemm_smallm(df.gate_up_swiglu_batched(rms_norm(x, n2, EPS), wgu), wd, residual=x)
    return x


def _exact(x, layers, size, cos, sin, n, rows_of):
    H, I, nq, nkv, D = SIZES[size]
    x = x[0].double()
    c, s = cos[n - 1].double(), sin[n - 1].double()

    def norm(v, w):
        return v * torch.rsqrt(v.square().mean() + EPS) * w.double()

    def turn(v):
        a, b = v.chunk(2, dim=-1)
        return torch.cat([a * c - b * s, b * c + a * s], dim=-1)

    for n1, wqkv, wo, n2, wgu, wd, ck, cv in layers:
        q, k, v = (wqkv.double() @ norm(x, n1)).reshape(-1, D).split([nq, nkv, nkv])
        keys = torch.cat([rows_of(ck)[:, :n - 1].double(), turn(k).unsqueeze(1)], dim=1)
        values = torch.cat([rows_of(cv)[:, :n - 1].double(), v.unsqueeze(1)], dim=1)
        p = torch.softmax(torch.einsum("ghd,gnd->ghn", turn(q).reshape(nkv, -1, D), keys) * D ** -0.5, dim=-1)
        x = x + wo.double() @ torch.einsum("ghn,gnd->ghd", p, values).flatten()
        g, u = (wgu.double() @ norm(x, n2)).chunk(2)
        x = x + wd.double() @ (torch.nn.functional.silu(g) * u)
    return x


def _stack(x, layers, size, cos, sin, pos, lens, **place):
    from neuronx_distributed_llama3_2_b200.ops import decode_fused as df

    H, I, nq, nkv, D = SIZES[size]
    scratch = df.token_stack_scratch(len(layers), 1, H, I, nq, nkv, D)
    assert scratch > 0 and df.token_stack_scratch(len(layers), 2, H, I, nq, nkv, D) == 0
    return df.token_stack(x, [(tuple(w), EPS, EPS) for w in layers], cos, sin, pos, lens, nq, nkv, D, scratch, **place)


@pytest.mark.parametrize("size", SIZES)
# the first token, edges of the parts of 256 keys, of the ring's slots of 64 and 128 keys, more keys than 16 parts of 256; pages that end inside a
# slot and hold whole ones; as many keys that a CTA's share goes through the ring of six slots once (12.5 and 6.5 thousand), three and ten
# times, in 16 and 18 parts
@pytest.mark.parametrize("n,page", [(1, 0), (2, 16), (64, 0), (257, 128), (511, 16), (4500, 128), (6500, 0), (12500, 16), (20000, 128), (40000, 0),
                                    (65536, 128), (65537, 0), (131072, 0)])
def test_layers_in_one_launch(size, n, page):
    H, I, nq, nkv, D = SIZES[size]
    lines, rows = 2, (n + 127) // 128 * 128
    layers, x = _draw(size, 2, lines, rows, n)
    cos, sin = _tables(D, rows)
    place = {"seq_ids": torch.tensor([1], dtype=torch.int32, device="cuda")}

    def rows_of(cache):
        return cache[1]

    if page:
        order = torch.randperm(lines * rows // page, generator=torch.Generator().manual_seed(n)).cuda()
        place.update(block_table=order.to(torch.int32).reshape(lines, -1), page_size=page)
        for w in layers:
            w[6:] = [t.reshape(-1, nkv, page, D) for t in w[6:]]

        def rows_of(cache):
            return cache[order.reshape(lines, -1)[1]].transpose(0, 1).flatten(1, 2)

    pos, lens = (torch.tensor([v], dtype=torch.int32, device="cuda") for v in (n - 1, n))
    ref = _exact(x, layers, size, cos, sin, n, rows_of)
    other = [[t.clone() for t in w] for w in layers]
    chain = _chain(x, other, size, cos, sin, pos, lens, **place)
    before = [[rows_of(t).clone() for t in w[6:]] for w in layers]
    out = _stack(x, layers, size, cos, sin, pos, lens, **place)

    def off(y):
        return float((y[0].double() - ref).norm() / ref.norm())

    assert off(out) <= 1.25 * off(chain)          # the same roundings of other sums: 0.97 to 1.03 times as far off
    for w, c, b in zip(layers, other, before):
        for mine, theirs, was in zip(w[6:], c[6:], b):
            mine, theirs = rows_of(mine), rows_of(theirs)
            assert torch.equal(mine[:, :n - 1], was[:, :n - 1]) and torch.equal(mine[:, n:], was[:, n:])
            # projections of streams that differ by a few roundings to bf16
            assert (mine[:, n - 1].float() - theirs[:, n - 1].float()).norm() <= 2e-2 * theirs[:, n - 1].float().norm()
    for _ in range(3 if n > 6000 else 1):
        assert torch.equal(out, _stack(x, layers, size, cos, sin, pos, lens, **place))


@pytest.mark.parametrize("size", SIZES)
def test_a_value_that_is_not_finite_stays_in_its_channel(size):
    H, I, nq, nkv, D = SIZES[size]
    layers, x = _draw(size, 1, 1, 128, 3)
    for i, row in ((5, float("inf")), (D + D // 2 + 2, float("nan"))):                 # of the value heads: a lower and an upper half
        layers[0][1][(nq + nkv) * D + i] = row
    cos, sin = _tables(D, 128)
    pos, lens = (torch.tensor([v], dtype=torch.int32, device="cuda") for v in (99, 100))
    other = [[t.clone() for t in w] for w in layers]
    _chain(x, other, size, cos, sin, pos, lens)
    _stack(x, layers, size, cos, sin, pos, lens)
    (ck, cv), (k, v) = layers[0][6:], other[0][6:]
    finite = torch.isfinite(cv[0, :, 99])
    assert torch.equal(finite, torch.isfinite(v[0, :, 99])) and (~finite).sum() == 2 and torch.isfinite(ck).all()
    assert (cv[0, :, 99][finite].float() - v[0, :, 99][finite].float()).norm() <= 2e-2 * v[0, :, 99][finite].float().norm()     # as above


def test_replays_follow_the_position():
    H, I, nq, nkv, D = SIZES["64"]
    layers, x = _draw("64", 2, 1, 640, 7)
    cos, sin = _tables(D, 640)
    pos, lens = (torch.tensor([v], dtype=torch.int32, device="cuda") for v in (300, 301))
    run = [[t.clone() for t in w] for w in layers]
    _stack(x, run, "64", cos, sin, pos, lens)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = _stack(x, run, "64", cos, sin, pos, lens)
    for n in (301, 302, 20, 600):
        pos.fill_(n - 1)
        lens.fill_(n)
        for w, given in zip(run, layers):
            for mine, theirs in zip(w[6:], given[6:]):
                mine.copy_(theirs)
        graph.replay()
        eager = [[t.clone() for t in w] for w in layers]
        assert torch.equal(out, _stack(x, eager, "64", cos, sin, pos, lens))
        assert all(torch.equal(a, b) for w, e in zip(run, eager) for a, b in zip(w[6:], e[6:]))


def test_waits_give_up():
    """Limits from none at all up to more than a step takes: what is left is the result or NaN, and the host is told."""
    from neuronx_distributed_llama3_2_b200.ops import decode_fused as df

    H, I, nq, nkv, D = SIZES["64"]
    layers, x = _draw("64", 2, 1, 256, 9)
    cos, sin = _tables(D, 256)
    pos, lens = (torch.tensor([v], dtype=torch.int32, device="cuda") for v in (99, 100))
    df.token_stack_gave_up()
    good = _stack(x, layers, "64", cos, sin, pos, lens)
    assert not df.token_stack_gave_up() and torch.isfinite(good).all()
    for clocks in (0, 100, 1000, 10000, 100000, -1):
        out = _stack(x, layers, "64", cos, sin, pos, lens, wait_clocks=clocks)
        gave_up = df.token_stack_gave_up()
        assert (out.isnan() | (out == good)).all() and (gave_up or not out.isnan().any())
        if clocks == 0:
            assert gave_up and out.isnan().all()
        if clocks == -1:
            assert not gave_up


def _model(cls=None, lines=1, **cache):
    """Two layers of the 2048-wide model with a small vocabulary."""
    from neuronx_distributed_llama3_2_b200.inference import InferenceConfig, LlamaInferenceModel
    from neuronx_distributed_llama3_2_b200.models import LlamaConfig

    H, I, nq, nkv, D = SIZES["64"]
    torch.manual_seed(11)
    cfg = LlamaConfig(vocab_size=512, hidden_size=H, intermediate_size=I, num_hidden_layers=2, num_attention_heads=nq, num_key_value_heads=nkv)
    model = (cls or LlamaInferenceModel)(cfg, InferenceConfig(batch_size=lines, max_context_length=64, seq_len=256, **cache),
                                         device=torch.device("cuda"))
    model.init_kv_cache(device=torch.device("cuda"))
    return model


def test_a_step_that_gave_up_reaches_the_program():
    from neuronx_distributed_llama3_2_b200.inference.model_builder import BaseModelInstance, ModelBuilder

    model = _model()
    ids = torch.randint(1, 512, (1, 20), device="cuda")
    good = model.generate(ids, max_new_tokens=6)
    tok, pos = ids[:, :1], torch.full((1, 1), 20, device="cuda")
    model._token_stack_clocks = 0                        # every wait gives up at once
    model.forward_infer(tok, pos)
    torch.cuda.synchronize()
    model._token_stack_clocks = -1
    with pytest.raises(RuntimeError, match="gave up"):
        model.forward_infer(tok, pos)
    model.forward_infer(tok, pos)                        # told once
    model._token_stack_clocks = 0
    with pytest.raises(RuntimeError, match="gave up"):
        model.generate(ids, max_new_tokens=2)
    model._token_stack_clocks = -1
    assert torch.equal(model.generate(ids, max_new_tokens=6), good)
    model.check_steps()
    copy.deepcopy(model).check_steps()
    with torch.device("cuda"):                           # the word is host memory whatever the default device is
        copy.deepcopy(model).init_kv_cache()
    graph = torch.cuda.CUDAGraph()                       # a replay asks nobody: the word is there behind it
    model._token_stack_clocks = 0
    with torch.cuda.graph(graph):
        model.forward_infer(tok, pos)
    model.check_steps()
    graph.replay()
    torch.cuda.synchronize()
    with pytest.raises(RuntimeError, match="gave up"):
        model.check_steps()
    model._token_stack_clocks = -1
    traced = ModelBuilder().add("token", BaseModelInstance(lambda: model), [(tok, pos)]).trace(initialize_model_weights=False)
    traced(tok, pos)
    model._gave_up.word.fill_(1)
    with pytest.raises(RuntimeError, match="gave up"):
        traced(tok, pos)
    traced(tok, pos)


def test_a_stream_of_fewer_multiprocessors_takes_the_layers_one_by_one():
    """One launch needs every SM of the device at once; in a green context of half of them the chain of kernels runs, as it always did."""
    from torch.cuda.green_contexts import SUPPORTED, GreenContext

    if not SUPPORTED:
        pytest.skip("this torch has no green contexts")
    from neuronx_distributed_llama3_2_b200.ops import decode_fused as df

    model = _model()
    tok, pos = torch.full((1, 1), 5, device="cuda"), torch.zeros((1, 1), dtype=torch.long, device="cuda")
    assert df.token_stack_runs_here()
    stacked = model.forward_infer(tok, pos, return_logits=True)[1]
    torch.cuda.synchronize()
    some = GreenContext.create(64, 0)
    some.set_context()
    try:
        here = df.token_stack_runs_here()
        chain = model.forward_infer(tok, pos, return_logits=True)[1]
        torch.cuda.synchronize()
    finally:
        some.pop_context()
    assert not here
    assert (stacked - chain).float().norm() <= 4e-2 * chain.float().norm()       # two layers, rounded to bf16 at the same places


def _counted(model, monkeypatch):
    """How often the model's layers ran in one launch."""
    from neuronx_distributed_llama3_2_b200.ops import decode_fused as df

    calls, real = [], df.token_stack
    monkeypatch.setattr(df, "token_stack", lambda *a, **k: calls.append(1) or real(*a, **k))
    return calls


def test_what_a_program_puts_in_the_place_of_a_step_is_called(monkeypatch):
    from neuronx_distributed_llama3_2_b200.inference import LlamaInferenceModel

    class Own(LlamaInferenceModel):
        def _decode_attention(self, q, ck, cv, seq_ids, lengths):
            return torch.zeros_like(q)

    tok, pos = torch.full((1, 1), 5, device="cuda"), torch.zeros((1, 1), dtype=torch.long, device="cuda")
    own = _model(Own).forward_infer(tok, pos, return_logits=True)[1]
    model = _model()
    calls = _counted(model, monkeypatch)
    model._decode_attention = lambda q, ck, cv, seq_ids, lengths: torch.zeros_like(q)
    assert torch.equal(model.forward_infer(tok, pos, return_logits=True)[1], own) and not calls
    del model._decode_attention
    assert not torch.equal(model.forward_infer(tok, pos, return_logits=True)[1], own) and len(calls) == 1


@pytest.mark.parametrize("kind", ["contiguous", "paged", "lines", "paged lines"])
def test_the_model_takes_it(kind, monkeypatch):
    """Order and shape of the weights, cache lines and pages: against the same model's layers kernel by kernel."""
    model = _model(lines=3, paged_kv="paged" in kind, page_size=16, is_continuous_batching="lines" in kind)
    gen = torch.Generator(device="cuda").manual_seed(2)
    ids = torch.randint(1, 512, (3, 40), generator=gen, device="cuda")
    pos = torch.arange(40, device="cuda").unsqueeze(0).expand(3, 40)
    lines = torch.arange(3, dtype=torch.int32, device="cuda")
    model.forward_infer(ids, pos, seq_ids=lines)
    saved = [t.clone() for t in model.kv_cache.k + model.kv_cache.v]
    line = lines[2:] if "lines" in kind else None
    step = (ids[:1, :1], torch.full((1, 1), 40, device="cuda"), line)
    calls = _counted(model, monkeypatch)
    stacked = model.forward_infer(*step, return_logits=True)[1]
    assert len(calls) == 1
    mine = [t.clone() for t in model.kv_cache.k + model.kv_cache.v]
    for t, was in zip(model.kv_cache.k + model.kv_cache.v, saved):
        t.copy_(was)
    with monkeypatch.context() as m:
        m.setattr(model, "_token_stack", lambda *_: None)
        chain = model.forward_infer(*step, return_logits=True)[1]
    assert len(calls) == 1
    # two layers, every value rounded to bf16 at the same places: 2^-8 of a vector each, some ten of them on the way
    assert (stacked - chain).float().norm() <= 4e-2 * chain.float().norm()
    for a, b, was in zip(mine, model.kv_cache.k + model.kv_cache.v, saved):
        changed = (b != was).any(-1)                     # one row per key head, of that line
        assert torch.equal((a != was).any(-1), changed) and changed.sum() == 8
        assert (a[changed].float() - b[changed].float()).norm() <= 2e-2 * b[changed].float().norm()
    other = lines[:1] if "lines" in kind else None
    if other is not None:                                # another line, another context
        assert not torch.equal(model.forward_infer(step[0], step[1], other, return_logits=True)[1], stacked)


def test_the_model_leaves_other_steps_alone(monkeypatch):
    model = _model(lines=2)
    calls = _counted(model, monkeypatch)
    two = torch.full((2, 1), 5, device="cuda"), torch.zeros((2, 1), dtype=torch.long, device="cuda")
    one = two[0][:1], two[1][:1]
    model.forward_infer(*two)                                                  # two sequences
    model.forward_infer(torch.full((1, 4), 5, device="cuda"), torch.arange(4, device="cuda").unsqueeze(0))      # a prompt
    assert not calls
    model.forward_infer(*one)
    assert len(calls) == 1
    norm = model.model.layers[1].post_attention_layernorm
    norm.weight.data = norm.weight.data.float()                                # a norm that is kept in fp32
    assert torch.isfinite(model.forward_infer(*one, return_logits=True)[1]).all() and len(calls) == 1
