"""Retention of long steps on the tensor cores, against float64 token by token."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _turn(x, pos, cos, sin, layout):
    rot = 2 * cos.shape[1]
    c, s = cos[pos].double().unsqueeze(-2), sin[pos].double().unsqueeze(-2)
    y = x.clone()
    if layout == "halves":
        u, v = x[..., : rot // 2], x[..., rot // 2: rot]
        y[..., : rot // 2], y[..., rot // 2: rot] = u * c - v * s, v * c + u * s
    else:
        u, v = x[..., 0:rot:2], x[..., 1:rot:2]
        y[..., 0:rot:2], y[..., 1:rot:2] = u * c - v * s, v * c + u * s
    return y


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
# steps around the 256-token chunk, ragged and empty rows; sizes around the 64-term blocks and the 128-column tiles
@pytest.mark.parametrize("T,n_new", [(128, None), (257, [257, 1, 0]), (600, [511, 600, 513])])
@pytest.mark.parametrize("H,D,Dv,rot,layout", [(3, 64, 64, 64, "halves"), (2, 128, 192, 96, "pairs"), (1, 256, 512, 256, "halves"),
                                               (2, 192, 128, 0, "halves"), (2, 64, 128, 64, "halves")])
def test_long_steps_match_float64(dtype, T, n_new, H, D, Dv, rot, layout, monkeypatch):
    from neuronx_distributed_llama3_2_b200.ops import retention as ret

    monkeypatch.setattr(ret, "_tc_wanted", lambda *sizes: True)          # the smallest states are faster on the fp32 kernels

    B, lines = 3, 4
    gen = torch.Generator(device="cuda").manual_seed(T + D)
    line = torch.tensor([2, 0, 3], dtype=torch.int32, device="cuda")
    decay = torch.tensor([0.9995, 0.3, 0.97], device="cuda")[:H]
    state = torch.randn(lines, H, D, Dv, generator=gen, device="cuda")
    ang = torch.outer(torch.arange(2 * T, dtype=torch.float64), 0.7 ** torch.arange(rot // 2, dtype=torch.float64))
    cos, sin = ang.cos().float().cuda(), ang.sin().float().cuda()
    at, states = [0] * B, [None] * B
    for _ in range(2):                                   # a prompt, then a portion that continues its state
        proj = torch.randn(B, T, 2 * H * D + H * Dv + 24, generator=gen, device="cuda").to(dtype)
        new = None if n_new is None else torch.tensor(n_new, dtype=torch.int32, device="cuda")
        before = state.clone()
        out = ret.retention_chunkwise(proj, (8, 8 + H * D, 16 + 2 * H * D), decay, state,
                                      torch.tensor(at, dtype=torch.int32, device="cuda"), H, D, Dv, D ** -0.5,
                                      (cos, sin) if rot else None, layout, n_new=new, seq_ids=line)
        assert torch.equal(state[1], before[1])
        for b in range(B):
            n = T if n_new is None else n_new[b]
            assert not out[b, n:].any()
            if n == 0:
                assert torch.equal(state[line[b]], before[line[b]])
                continue
            x = proj[b, :n].double()
            q, k = (x[:, o: o + H * D].unflatten(-1, (H, D)) for o in (8, 8 + H * D))
            v = x[:, 16 + 2 * H * D: 16 + 2 * H * D + H * Dv].unflatten(-1, (H, Dv))
            if rot:
                pos = torch.arange(at[b], at[b] + n, device="cuda")
                q, k = (_turn(y, pos, cos, sin, layout) for y in (q, k))
            k = k * D ** -0.5
            S = torch.zeros(H, D, Dv, dtype=torch.float64, device="cuda") if at[b] == 0 else states[b]
            ref = torch.empty(n, H, Dv, dtype=torch.float64, device="cuda")
            a = decay.double().reshape(H, 1, 1)
            for t in range(n):
                S = a * S + k[t].unsqueeze(-1) * v[t].unsqueeze(-2)
                ref[t] = torch.einsum("hdv,hd->hv", S, q[t])
            states[b] = S
            at[b] += n
            # 64-term sums on the tensor cores are off by 7e-8, twice in a row for the scores' share; the kernel's powers of
            # the decay and the rotation add a few roundings of 6e-8
            assert (out[b, :n] - ref).norm() <= 3e-7 * ref.norm()
            assert (state[line[b]] - S).norm() <= 3e-7 * S.norm()


def test_a_value_that_is_not_a_number_leaves_the_tokens_before_it_alone():
    from neuronx_distributed_llama3_2_b200.ops import retention as ret

    T, H, D, Dv = 600, 1, 64, 128
    gen = torch.Generator(device="cuda").manual_seed(1)
    clean = torch.randn(1, T, 2 * D + Dv, generator=gen, device="cuda")
    decay, start = torch.tensor([0.9], device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")

    def run(proj):
        S = torch.zeros(1, H, D, Dv, device="cuda")
        return ret.retention_chunkwise(proj, (0, D, 2 * D), decay, S, start, H, D, Dv)[0, :, 0], S[0, 0]

    good, good_S = run(clean)
    for where, token, column in (("value", 300, 5), ("key", 300, 7), ("query", 300, 7)):
        proj = clean.clone()
        proj[0, token, {"query": 0, "key": D, "value": 2 * D}[where] + column] = float("nan")
        out, S = run(proj)
        assert torch.equal(out[:token], good[:token])
        if where == "value":
            others = torch.arange(Dv, device="cuda") != column
            assert out[token:, column].isnan().all() and S[:, column].isnan().all()
            assert torch.equal(out[:, others], good[:, others]) and torch.equal(S[:, others], good_S[:, others])
        elif where == "key":
            assert out[token:].isnan().all() and S[column].isnan().all()
        else:
            assert out[token].isnan().all() and torch.equal(out[token + 1:], good[token + 1:]) and torch.equal(S, good_S)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
# rotations of whole vectors, of parts of one and of neighbours; rows, values and tables that take 16-byte loads and ones that do not
@pytest.mark.parametrize("D,rot,layout", [(64, 48, "halves"), (64, 40, "halves"), (128, 24, "pairs"), (64, 64, "pairs"), (256, 32, "halves")])
@pytest.mark.parametrize("first", [0, 3])
def test_rotations_and_rows_at_odd_addresses(dtype, D, rot, layout, first, monkeypatch):
    from neuronx_distributed_llama3_2_b200.ops import retention as ret

    monkeypatch.setattr(ret, "_tc_wanted", lambda *sizes: True)
    T, H, Dv = 67, 2, 64
    gen = torch.Generator(device="cuda").manual_seed(D + rot)
    proj = torch.randn(1, T, 2 * H * D + H * Dv + first, generator=gen, device="cuda").to(dtype)
    ang = torch.outer(torch.arange(T, dtype=torch.float64), 0.7 ** torch.arange(rot // 2, dtype=torch.float64))
    tables = torch.stack([ang.cos(), ang.sin()]).float().cuda()
    decay, S = torch.tensor([0.98, 0.9], device="cuda"), torch.zeros(1, H, D, Dv, device="cuda")
    out = ret.retention_chunkwise(proj, (first, first + H * D, first + 2 * H * D), decay, S,
                                  torch.zeros(1, dtype=torch.int32, device="cuda"), H, D, Dv, D ** -0.5, tuple(tables), layout)[0]
    q, k, v = proj[0, :, first:].double().split([H * D, H * D, H * Dv], dim=-1)
    q, k = (_turn(x.unflatten(-1, (H, D)), torch.arange(T, device="cuda"), *tables, layout) for x in (q, k))
    t = torch.arange(T, dtype=torch.float64, device="cuda")
    for h in range(H):
        scores = (q[:, h] @ k[:, h].t() * D ** -0.5 * decay[h].double() ** (t.unsqueeze(1) - t).clamp(min=0)).tril()
        ref = scores @ v.unflatten(-1, (H, Dv))[:, h]
        assert (out[:, h] - ref).norm() <= 3e-7 * ref.norm()             # as above
