"""The recurrences over prompts, sixteen tokens at a time: lengths around a chunk's edge against 64-bit arithmetic token after token,
and an infinity or a NaN in one token, which must not reach the tokens in front of it, other columns or other sequences."""
import pytest
import torch

from test_gpu_recurrent_chunks import DEV, batch, both_ways, off

pytestmark = pytest.mark.gpu


def delta_inputs(T, G, D, H, V, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    qk = torch.randn((T, 2 * G, D), generator=g, device=DEV)
    qk = qk / qk.norm(dim=-1, keepdim=True)
    qkv = torch.cat([qk.flatten(1), torch.randn((T, H * V), generator=g, device=DEV)], 1).contiguous()
    beta = torch.sigmoid(torch.randn((T, H), generator=g, device=DEV))
    decay = torch.exp(-torch.rand((T, H), generator=g, device=DEV) * 0.1)
    return qkv, beta, decay, g


def delta_call(qkv, beta, decay, G, D, H, V, view):
    from inference_engine_rust_b200.csrc import bindings as B
    T = qkv.shape[0]

    def call(s):
        o = torch.zeros((T, H * V), device=DEV)
        scratch = torch.full((B.recurrent_scratch_floats(D, T, H),), float("nan"), device=DEV)
        B.delta_recur(qkv, beta, decay, s, 0, o, G, D, H, V, view, B.stream_ptr(), scratch=scratch)
        return o
    return call


@pytest.mark.parametrize("D,V,H,G", [(128, 128, 10, 1), (64, 44, 3, 1)])      # (ten heads share a key head; a rest of 12 columns)
@pytest.mark.parametrize("lens", [[31], [32], [33], [17, 16, 48, 47, 15]])
def test_delta_rule_at_a_chunks_edge(monkeypatch, D, V, H, G, lens):
    T, n = sum(lens), len(lens)
    qkv, beta, decay, g = delta_inputs(T, G, D, H, V, T + D)
    state = torch.randn((n, H * D * V), generator=g, device=DEV)
    view, keep = batch(lens, list(range(n)))
    (o, s), (o1, s1) = both_ways(monkeypatch, delta_call(qkv, beta, decay, G, D, H, V, view), state)
    q, k, v = (x.double() for x in (qkv[:, :G * D].view(T, G, D), qkv[:, G * D:2 * G * D].view(T, G, D), qkv[:, 2 * G * D:].view(T, H, V)))
    q, k = (x.repeat_interleave(H // G, 1) for x in (q, k))
    want_o, want_s, at = torch.zeros((T, H, V), dtype=torch.float64, device=DEV), state.double().view(n, H, D, V).clone(), 0
    for i, m in enumerate(lens):
        S = want_s[i]
        for t in range(at, at + m):
            S *= decay[t].double()[:, None, None]
            u = beta[t].double()[:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t]))
            S += k[t][:, :, None] * u[:, None]
            want_o[t] = torch.einsum("hdv,hd->hv", S, q[t])
        at += m
    for got, plain, want in ((o, o1, want_o.flatten(1)), (s, s1, want_s.flatten(1))):
        # sums of up to DIM + 16 terms, rounded to 2^-24 each, as in the kernel that goes token after token
        assert off(got, want) <= 2.0 ** -20
        assert off(got, want) <= 1.25 * off(plain, want) + 2.0 ** -25


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("at", [16, 21, 31])
def test_delta_rule_keeps_a_lost_number_in_its_place(monkeypatch, bad, at):
    G, D, H, V, lens = 1, 128, 2, 64, [48, 32]
    qkv, beta, decay, g = delta_inputs(80, G, D, H, V, 5)
    state = torch.randn((2, H * D * V), generator=g, device=DEV)
    view, keep = batch(lens, [0, 1])
    whole = delta_call(qkv, beta, decay, G, D, H, V, view)(state.clone()).view(80, H, V)
    qkv = qkv.clone()
    qkv[at, 2 * G * D + V + 37] = bad                              # head 1, column 37
    (o, _), (o1, _) = both_ways(monkeypatch, delta_call(qkv, beta, decay, G, D, H, V, view), state)
    o, o1 = o.view(80, H, V), o1.view(80, H, V)
    assert torch.equal(torch.isfinite(o), torch.isfinite(o1))
    touched = torch.zeros_like(whole, dtype=torch.bool)
    touched[at:48, 1, 37] = True
    # in front of it the sums are formed another way (plain multiply-adds); everything else is as without it
    rest = ~touched
    rest[16:48, 1] = False
    assert torch.equal(o[rest], whole[rest])
    near = 2.0 ** -20 * whole.abs().max().item()                    # two sums of D + 16 rounded terms, in another order
    others = [c for c in range(V) if c != 37]
    assert (o[16:48, 1][:, others] - whole[16:48, 1][:, others]).abs().max().item() <= near
    if at > 16:
        assert (o[16:at, 1, 37] - whole[16:at, 1, 37]).abs().max().item() <= near


@pytest.mark.parametrize("lens", [[48], [63], [65], [17, 16, 112, 47, 100]])
def test_decay_per_key_channel_at_a_chunks_edge(monkeypatch, lens):
    from inference_engine_rust_b200.csrc import bindings as B
    D, V, H, T, n = 64, 44, 3, sum(lens), len(lens)
    g = torch.Generator(device=DEV).manual_seed(T)
    x = torch.randn((T, 2 * H * D + H * V), generator=g, device=DEV)
    decay = torch.exp(-torch.exp(torch.rand((T, H * D), generator=g, device=DEV) * 6 - 6))
    u = torch.randn((H, D), generator=g, device=DEV)
    state = torch.randn((n, H * D * V), generator=g, device=DEV)
    view, keep = batch(lens, list(range(n)))

    def call(s, xx=x):
        o = torch.zeros((T, H * V), device=DEV)
        scratch = torch.full((B.recurrent_scratch_floats(D, T, H),), float("nan"), device=DEV)
        B.wkv_recur(xx, decay, u, s, 0, o, D, H, V, view, B.stream_ptr(), scratch=scratch)
        return o
    (o, s), (o1, s1) = both_ways(monkeypatch, call, state)
    r, k, v = (x[:, a:b].double().view(T, H, -1) for a, b in ((0, H * D), (H * D, 2 * H * D), (2 * H * D, 2 * H * D + H * V)))
    w = decay.double().view(T, H, D)
    want_o, want_s, at = torch.zeros((T, H, V), dtype=torch.float64, device=DEV), state.double().view(n, H, D, V).clone(), 0
    for i, m in enumerate(lens):
        S = want_s[i].clone()
        for t in range(at, at + m):
            kv = k[t][:, :, None] * v[t][:, None]
            want_o[t] = torch.einsum("hdv,hd->hv", S + u.double()[:, :, None] * kv, r[t])
            S = S * w[t][:, :, None] + kv
        want_s[i] = S
        at += m
    for got, plain, want in ((o, o1, want_o.flatten(1)), (s, s1, want_s.flatten(1))):
        assert off(got, want) <= 2.0 ** -20
        assert off(got, want) <= 1.25 * off(plain, want) + 2.0 ** -25
    # a NaN in one value stays in its column, behind its token, in its sequence
    bad, t = x.clone(), min(20, lens[0] - 1)
    bad[t, 2 * H * D + V + 37] = float("nan")
    got = call(state.clone(), bad).view(T, H, V)
    lost = torch.zeros((T, H, V), dtype=torch.bool, device=DEV)
    lost[t:lens[0], 1, 37] = True
    assert torch.equal(torch.isnan(got), lost)
    # two sums of D + 16 rounded terms, in another order
    assert (got - o.view(T, H, V))[~lost].abs().max().item() <= 2.0 ** -20 * o.abs().max().item()
