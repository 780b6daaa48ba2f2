"""Chunk-wise gated delta rule and the strip-wise short convolution ahead of it, against float64 token by token."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _oracle(q, k, v, g, beta, S):
    """q, k [T, G, D], v [T, H, Dv], g, beta [T, H], S [H, D, Dv]."""
    H, rep = v.shape[1], v.shape[1] // q.shape[1]
    out = []
    for t in range(q.shape[0]):
        kt, qt = (x[t].repeat_interleave(rep, dim=0) for x in (k, q))
        S = S * g[t].reshape(H, 1, 1)
        u = beta[t].reshape(H, 1) * (v[t] - torch.einsum("hdv,hd->hv", S, kt))
        S = S + kt.unsqueeze(-1) * u.unsqueeze(1)
        out.append(torch.einsum("hdv,hd->hv", S, qt))
    return torch.stack(out), S


# steps around the 64-token chunk, ragged and empty rows, a second portion that continues the state; decays from none to total
@pytest.mark.parametrize("D,H,G,Dv", [(64, 2, 2, 32), (64, 4, 2, 96), (128, 2, 1, 256), (256, 1, 1, 64)])
@pytest.mark.parametrize("T,n_new", [(192, None), (257, [257, 1, 0]), (200, [129, 200, 64])])
@pytest.mark.parametrize("strength", [-6.0, 0.0, 6.0])
def test_chunks_match_float64(D, H, G, Dv, T, n_new, strength):
    from neuronx_distributed_llama3_2_b200.ops import delta_rule as dr

    B, lines = 3, 4
    gen = torch.Generator(device="cuda").manual_seed(D + T)

    def normal(*s):
        return torch.randn(*s, generator=gen, device="cuda")

    line = torch.tensor([2, 0, 3], dtype=torch.int32, device="cuda")
    S = normal(lines, H, D, Dv)
    a_log, dt_bias = normal(H) * 0.5 + strength, normal(H)
    states, at = [None] * B, [0] * B
    for _ in range(2):
        q = F.normalize(normal(B, T, G, D), dim=-1) * D ** -0.5
        k, v = F.normalize(normal(B, T, G, D), dim=-1), normal(B, T, H, Dv)
        a_pre, b_pre = normal(B * T, H + 3), normal(B * T, H + 1)
        new = None if n_new is None else torch.tensor(n_new, dtype=torch.int32, device="cuda")
        g = torch.exp(-torch.exp(a_log.double()) * F.softplus(a_pre[:, 3:].double() + dt_bias.double())).reshape(B, T, H)
        beta = torch.sigmoid(b_pre[:, 1:].double()).reshape(B, T, H)
        before = S.clone()
        out = dr.delta_scan(q, k, v, a_pre, 3, b_pre, 1, a_log, dt_bias, S, torch.tensor(at, dtype=torch.int32, device="cuda"),
                            False, n_new=new, seq_ids=line)
        assert torch.equal(S[1], before[1])              # a line that no row uses
        for b in range(B):
            n = T if n_new is None else n_new[b]
            assert not out[b, n:].any()
            if n == 0:
                assert torch.equal(S[line[b]], before[line[b]])
                continue
            start = torch.zeros(H, D, Dv, dtype=torch.float64, device="cuda") if at[b] == 0 else states[b]
            ref, states[b] = _oracle(q[b, :n].double(), k[b, :n].double(), v[b, :n].double(), g[b, :n], beta[b, :n], start)
            at[b] += n
            # per token a few roundings of 2^-24 (6e-8), each of which fades with the decay: the sums of exponentials that make
            # g are off by 1e-7 of the decay's distance from one per step, which weak decays collect over all tokens so far
            bound = (at[b] if strength < 0 else 8) ** 0.5 * 3e-7
            assert (out[b, :n] - ref).norm() <= bound * ref.norm()
            assert (S[line[b]] - states[b]).norm() <= bound * states[b].norm()


# keys from independent to nearly parallel, decays and learning rates from ordinary to next to one: where neighbouring tokens
# overwrite one another, errors inside a chunk must not add up
@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("common,strength,rate", [(0.0, 0.0, 0.0), (0.6, -6.0, 4.0), (0.9, -4.0, 4.0), (0.97, -7.0, 6.0)])
def test_chunks_are_no_further_off_than_single_tokens(D, common, strength, rate):
    from neuronx_distributed_llama3_2_b200.ops import delta_rule as dr

    T, H, Dv, portion = 1024, 2, 64, 128                 # portions of 128 tokens run token by token
    gen = torch.Generator(device="cuda").manual_seed(D)

    def normal(*s):
        return torch.randn(*s, generator=gen, device="cuda")

    k, q = (F.normalize((1 - common) * normal(1, T, H, D) + common * x, dim=-1) for x in (normal(1, 1, H, D),) for _ in range(2))
    q, v = q * D ** -0.5, normal(1, T, H, Dv)
    a_pre, b_pre, start = normal(T, H), normal(T, H) + rate, normal(1, H, D, Dv)
    a_log, dt_bias = normal(H) * 0.1 + strength, normal(H)
    g = torch.exp(-torch.exp(a_log.double()) * F.softplus(a_pre.double() + dt_bias.double()))
    want, state = _oracle(q[0].double(), k[0].double(), v[0].double(), g, torch.sigmoid(b_pre.double()), start[0].double())

    def run(size):
        S, outs = start.clone(), []
        for t in range(0, T, size):
            at = torch.full((1,), t + 1, dtype=torch.int32, device="cuda")          # not at a sequence's start: S is read
            x, y, z = (r[:, t:t + size].contiguous() for r in (q, k, v))
            outs.append(dr.delta_scan(x, y, z, a_pre[t:t + size].clone(), 0, b_pre[t:t + size].clone(), 0, a_log, dt_bias, S, at, False))
        return (torch.cat(outs, 1)[0] - want).norm() / want.norm(), (S[0] - state).norm() / state.norm()

    # both forms are fp32: a quarter for the scatter of sums of roundings.  The state also takes the sum of a chunk's 64 errors u times
    # their keys: where it cancels, their roundings (2^-25 on average) do not, 8 x 2^-25 of a state that is about one u
    (out, S), (out_tokens, S_tokens) = run(T), run(portion)
    assert out <= 1.25 * out_tokens + 2.0 ** -24
    assert S <= 1.25 * S_tokens + 2.0 ** -22


# decays of a half and of a fifth per token: few tokens count, and every value is a handful of roundings -- of the factors, of U's and the
# state's three sums each, 2^-25.5 of a value on average: 6 + 2 of them in square 0.6e-7, a quarter more for the scatter
@pytest.mark.parametrize("strength", [0.0, 1.0])
@pytest.mark.parametrize("D", [64, 128, 256])
def test_chunks_with_strong_decays_are_off_by_their_last_roundings(D, strength):
    from neuronx_distributed_llama3_2_b200.ops import delta_rule as dr

    T, H, Dv = 640, 4, 128
    gen = torch.Generator(device="cuda").manual_seed(D)

    def normal(*s):
        return torch.randn(*s, generator=gen, device="cuda")

    q, k = (F.normalize(normal(1, T, H, D), dim=-1) for _ in range(2))
    q, v, S = q * D ** -0.5, normal(1, T, H, Dv), normal(1, H, D, Dv)
    g, beta, before = normal(T, H), normal(T, H), S[0].double()
    out = dr.delta_scan(q, k, v, g, 0, beta, 0, normal(H) * 0.1 + strength, normal(H) * 0.1, S,
                        torch.ones(1, dtype=torch.int32, device="cuda"), False)
    want, state = _oracle(q[0].double(), k[0].double(), v[0].double(), g.double(), beta.double(), before)     # the rounded gates
    assert (out[0] - want).norm() <= 1.25 * 2.0 ** -24 * want.norm()
    assert (S[0] - state).norm() <= 1.25 * 2.0 ** -24 * state.norm()


def test_a_token_that_is_not_a_number_leaves_the_tokens_before_it_alone():
    from neuronx_distributed_llama3_2_b200.ops import delta_rule as dr

    T, D, Dv = 192, 64, 32
    gen = torch.Generator(device="cuda").manual_seed(1)
    q, k = (F.normalize(torch.randn(1, T, 1, D, generator=gen, device="cuda"), dim=-1) for _ in range(2))
    v = torch.randn(1, T, 1, Dv, generator=gen, device="cuda")
    zero, start = torch.zeros(T, 1, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")

    def run(value):
        x = v.clone()
        x[0, 70, 0, 3] = value
        return dr.delta_scan(q, k, x, zero.clone(), 0, zero.clone(), 0, zero[0].clone(), zero[0].clone(),
                             torch.zeros(1, 1, D, Dv, device="cuda"), start, False)[0, :, 0]

    clean = run(0.5)
    for bad in (float("nan"), float("inf")):
        out = run(bad)
        assert torch.equal(out[:70], clean[:70]) and not torch.isfinite(out[70:, 3]).any()
    k[0, 69, 0, 5] = float("nan")                        # its row of the chunk's system
    assert torch.equal(run(0.5)[:69], clean[:69])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("D,H,G,Dv", [(64, 3, 1, 64), (128, 2, 2, 256), (256, 2, 1, 256)])
def test_strips_of_the_short_convolution_match_float64(dtype, D, H, G, Dv):
    from neuronx_distributed_llama3_2_b200.ops import delta_rule as dr

    B, taps, C = 2, 4, 2 * G * D + H * Dv
    gen = torch.Generator(device="cuda").manual_seed(D)
    long = 1 + 16 * (-(-1536 // (B * (2 * G + H * Dv // D))))        # enough of them for strips of 16
    total = 80 + long
    raw = torch.randn(B, total, C + 16, generator=gen, device="cuda").to(dtype)
    w = torch.randn(C, taps, generator=gen, device="cuda") * 0.5
    state = torch.randn(3, taps - 1, C, generator=gen, device="cuda")
    line = torch.tensor([2, 0], dtype=torch.int32, device="cuda")
    x = torch.cat([torch.zeros(B, taps - 1, C, dtype=torch.float64, device="cuda"), raw[..., 8:8 + C].double()], dim=1)
    act = F.silu(sum(w[:, j].double() * x[:, j:j + total] for j in range(taps)))
    q, k, v = act.split([G * D, G * D, H * Dv], dim=-1)
    q, k = (t.unflatten(-1, (G, D)) for t in (q, k))
    q, k = (t / torch.sqrt(t.square().sum(-1, keepdim=True) + 1e-6) for t in (q, k))
    refs = (q * 0.25, k, v.unflatten(-1, (H, Dv)))
    at = 0
    for size in (1, 17, 3, 16, 43, long):                # portions around the strips of 4 (few tokens) and 16
        got = dr.delta_prep(raw[:, at:at + size].contiguous(), (8, 8 + G * D, 8 + 2 * G * D), w, state,
                            torch.full((B,), at, dtype=torch.int32, device="cuda"), H, G, D, Dv, 0.25, seq_ids=line)
        for x32, ref in zip(got, refs):
            ref = ref[:, at:at + size]
            assert (x32 - ref).norm() <= 1e-6 * ref.norm()          # four products and a silu in fp32
        at += size
    assert torch.equal(state[line.long()], raw[:, -3:, 8:8 + C].float())


# operand tiles of half a gigabyte at most: eight rows of 32 heads take their seven chunks in two launches, a row alone in one
def test_steps_in_several_launches_are_the_same():
    from neuronx_distributed_llama3_2_b200.ops import delta_rule as dr

    B, T, H, D, Dv = 8, 421, 32, 256, 32
    gen = torch.Generator(device="cuda").manual_seed(2)

    def normal(*s):
        return torch.randn(*s, generator=gen, device="cuda")

    q, k = (F.normalize(normal(B, T, H, D), dim=-1) for _ in range(2))
    v, a_pre, b_pre, S = normal(B, T, H, Dv), normal(B * T, H), normal(B * T, H), normal(B, H, D, Dv)
    a_log, dt_bias = normal(H) - 2, normal(H)
    start = torch.ones(B, dtype=torch.int32, device="cuda")
    new = torch.tensor([T, 400, 384, 385, 1, 0, 64, 200], dtype=torch.int32, device="cuda")
    state = S.clone()
    out = dr.delta_scan(q, k, v, a_pre.clone(), 0, b_pre.clone(), 0, a_log, dt_bias, state, start, False, n_new=new)
    for b in range(B):
        rows, one = slice(b * T, (b + 1) * T), S[b:b + 1].clone()
        ref = dr.delta_scan(q[b:b + 1], k[b:b + 1], v[b:b + 1], a_pre[rows].clone(), 0, b_pre[rows].clone(), 0, a_log, dt_bias, one,
                            start[:1], False, n_new=new[b:b + 1])
        assert torch.equal(out[b], ref[0]) and torch.equal(state[b], one[0])


# limits from "at once" to "never": what gives up says so and leaves NaN behind its last good chunk, and the next call is sound
@pytest.mark.parametrize("D,Dv", [(64, 64), (128, 96), (256, 64)])
def test_a_wait_that_runs_out_is_reported(D, Dv):
    from neuronx_distributed_llama3_2_b200.ops import delta_rule as dr

    B, T, H = 2, 421, 3
    gen = torch.Generator(device="cuda").manual_seed(D)

    def normal(*s):
        return torch.randn(*s, generator=gen, device="cuda")

    q, k = (F.normalize(normal(B, T, H, D), dim=-1) for _ in range(2))
    v, a_pre, b_pre, S = normal(B, T, H, Dv), normal(B * T, H), normal(B * T, H), normal(B, H, D, Dv)
    a_log, dt_bias = normal(H) - 2, normal(H)
    start = torch.ones(B, dtype=torch.int32, device="cuda")

    def run(clocks):
        state = S.clone()
        out = dr._scan_on_gpu(q, k, v, a_pre.clone(), 0, b_pre.clone(), 0, a_log, dt_bias, state, start, False, wait_clocks=clocks)
        return out, state, dr.scan_gave_up()

    dr.scan_gave_up()
    out, state, gave_up = run(-1)
    assert not gave_up and torch.isfinite(state).all()
    for clocks in (0, 100, 1000, 10000, 100000, -1):
        x, s, gave_up = run(clocks)
        assert (s.isnan() | (s == state)).all() and (x.isnan() | (x == out)).all()
        assert gave_up or not (s.isnan().any() or x.isnan().any())
        assert gave_up != (clocks == -1) or 0 < clocks   # in between it depends on the clock
        if clocks == 0:
            assert s.isnan().all() and x.isnan().all()


# on either side of the lines between the scans: (row, head) pairs and tokens with one slice of 32 value columns and with two
@pytest.mark.parametrize("D,Dv,B,H,T,fp32", [(64, 32, 5, 19, 200, False), (64, 32, 3, 32, 200, True), (128, 32, 3, 32, 257, True),
                                             (256, 32, 8, 32, 192, False), (256, 32, 9, 32, 192, True), (64, 64, 4, 32, 320, True),
                                             (64, 64, 4, 32, 321, False), (64, 64, 16, 32, 385, True), (64, 96, 16, 32, 192, False)])
def test_both_scans_match_float64(D, Dv, B, H, T, fp32):
    from neuronx_distributed_llama3_2_b200.ops import _lib, delta_rule as dr

    gen = torch.Generator(device="cuda").manual_seed(D + Dv + B)

    def normal(*s):
        return torch.randn(*s, generator=gen, device="cuda")

    floats = _lib.lib().nxd_delta_scan_scratch(B, T, H, D, Dv, 0)
    assert (floats == B * H * -(-T // 64) * (2 * 64 * 64 + 2 * 64)) == fp32          # the fp32 scan has no operand tiles
    q, k = (F.normalize(normal(B, T, H, D), dim=-1) for _ in range(2))
    v, g, beta, S = normal(B, T, H, Dv), normal(B * T, H), normal(B * T, H), normal(B, H, D, Dv)
    new = [T, 130] + [T - b for b in range(2, B)]
    before = S.clone()
    out = dr.delta_scan(q, k, v, g, 0, beta, 0, normal(H) - 2, normal(H), S, torch.ones(B, dtype=torch.int32, device="cuda"), False,
                        n_new=torch.tensor(new, dtype=torch.int32, device="cuda"))
    for b in (0, 1, B - 1):
        n, rows = new[b], slice(b * T, b * T + new[b])
        want, state = _oracle(q[b, :n].double(), k[b, :n].double(), v[b, :n].double(), g[rows].double(), beta[rows].double(), before[b].double())
        # sums of fp32 roundings whose traces fade over some eight tokens: 8 ** 0.5 of the 2^-24 of one token
        assert (out[b, :n] - want).norm() <= 2.0 ** -22.5 * want.norm() and not out[b, n:].any()
        assert (S[b] - state).norm() <= 2.0 ** -22.5 * state.norm()


# operand tiles of more rows than half a gigabyte holds: rows in two launches, with and without lines of their own, each as it is alone
@pytest.mark.parametrize("lines", [False, True])
def test_rows_in_several_launches_are_the_same(lines):
    from neuronx_distributed_llama3_2_b200.ops import _lib, delta_rule as dr

    B, T, H, D, Dv = 25, 193, 64, 256, 64
    assert 4 * _lib.lib().nxd_delta_scan_scratch(B, T, H, D, Dv, 0) <= (512 << 20) * 11 // 10        # tiles and their systems
    gen = torch.Generator(device="cuda").manual_seed(3)

    def normal(*s):
        return torch.randn(*s, generator=gen, device="cuda")

    q, k = (F.normalize(normal(B, T, H, D), dim=-1) for _ in range(2))
    v, a_pre, b_pre, S = normal(B, T, H, Dv), normal(B * T, H), normal(B * T, H), normal(B + 1, H, D, Dv)
    a_log, dt_bias = normal(H) - 2, normal(H)
    start = (torch.arange(B, device="cuda") % 2).int()
    new = torch.tensor([T, 1, 0] + [T - b for b in range(3, B)], dtype=torch.int32, device="cuda")
    line = torch.randperm(B + 1, generator=gen, device="cuda")[:B].int() if lines else None
    state = S.clone()
    out = dr.delta_scan(q, k, v, a_pre.clone(), 0, b_pre.clone(), 0, a_log, dt_bias, state, start, False, n_new=new, seq_ids=line)
    for b in (0, 1, 2, 11, 12, 13, 14, B - 1):
        rows, at = slice(b * T, (b + 1) * T), int(line[b]) if lines else b
        one = S[at:at + 1].clone()
        ref = dr.delta_scan(q[b:b + 1], k[b:b + 1], v[b:b + 1], a_pre[rows].clone(), 0, b_pre[rows].clone(), 0, a_log, dt_bias, one,
                            start[b:b + 1], False, n_new=new[b:b + 1])
        assert torch.equal(out[b], ref[0]) and torch.equal(state[at], one[0])


# values, state and outputs that are not 16-byte aligned keep the chunks: where the fp32 scan serves anyway, bit for bit
@pytest.mark.parametrize("Dv,H,same", [(32, 48, True), (64, 4, False)])
def test_values_and_state_at_odd_addresses(Dv, H, same):
    from neuronx_distributed_llama3_2_b200.ops import delta_rule as dr

    B, T, D = 2, 200, 64
    gen = torch.Generator(device="cuda").manual_seed(4)

    def normal(*s):
        return torch.randn(*s, generator=gen, device="cuda")

    def odd(x):
        y = torch.empty(x.numel() + 1, device="cuda")[1:].view(x.shape)
        assert y.data_ptr() % 16 != 0
        return y.copy_(x)

    q, k = (F.normalize(normal(B, T, H, D), dim=-1) for _ in range(2))
    v, a_pre, b_pre, S = normal(B, T, H, Dv), normal(B * T, H), normal(B * T, H), normal(B, H, D, Dv)
    a_log, dt_bias, start = normal(H) - 2, normal(H), torch.ones(B, dtype=torch.int32, device="cuda")

    def run(v, S):
        return dr.delta_scan(q, k, v, a_pre.clone(), 0, b_pre.clone(), 0, a_log, dt_bias, S, start, False), S

    (x, s), (y, z) = run(v, S.clone()), run(odd(v), odd(S))
    if same:
        assert torch.equal(x, y) and torch.equal(s, z)
    # two scans, each within 2^-22.5 of float64
    assert (x - y).norm() <= 2.0 ** -21.5 * x.norm() and (s - z).norm() <= 2.0 ** -21.5 * s.norm()
