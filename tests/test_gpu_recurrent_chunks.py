"""The recurrences over prompts, eight tokens at a time: the gated delta rule and the recurrence with a decay per key channel
against 64-bit arithmetic token after token, at the edges of chunks and of the columns a block owns, from a state that is not
zero, with decays of 0 and 1; and no less precise than the kernels that go token after token."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
LENS = [40, 1, 7, 8, 9, 0, 33]          # 0: an empty sequence


def batch(lens, slots):
    from inference_engine_rust_b200.csrc import bindings as B
    n, T = len(lens), sum(lens)
    cu = torch.tensor([0] + lens).cumsum(0)
    arrs = [torch.as_tensor(a, dtype=torch.int32, device=DEV) for a in
            (cu, slots, torch.arange(n).repeat_interleave(torch.tensor(lens)), [0] * n)]
    view = B.BatchView(cu_q=arrs[0].data_ptr(), slot_ids=arrs[1].data_ptr(), tok_seq=arrs[2].data_ptr(), pos0=arrs[3].data_ptr(),
                       n_seqs=n, n_tokens=T)
    return view, arrs


def off(got, want):
    return ((got.double() - want).norm() / want.norm()).item()


def both_ways(monkeypatch, call, state):
    """(read-out, state) of the chunks and of the kernel that goes token after token."""
    out = []
    for lanes in (None, "16"):
        if lanes:
            monkeypatch.setenv("IERT_RECURRENT_LANES", lanes)
        s = state.clone()
        out.append((call(s), s))
        torch.cuda.synchronize()
        if lanes:
            monkeypatch.delenv("IERT_RECURRENT_LANES")
    return out


@pytest.mark.parametrize("D,V,H,G", [(128, 128, 4, 2), (64, 64, 3, 3), (128, 36, 2, 1), (64, 100, 4, 1)])
@pytest.mark.parametrize("lens", [LENS, [5], [2048], LENS + [100], [16], [15]])
def test_delta_rule(monkeypatch, D, V, H, G, lens):
    from inference_engine_rust_b200.csrc import bindings as B
    g = torch.Generator(device=DEV).manual_seed(D + V + len(lens))
    T, n, C = sum(lens), len(lens), 2 * G * D + H * V
    slots = list(range(n, 0, -1))
    slots[1 % n] = slots[1 % n] if n == 1 else -1                     # a padding sequence
    qk = torch.randn((T, 2 * G, D), generator=g, device=DEV)
    qk = qk / qk.norm(dim=-1, keepdim=True)
    qkv = torch.cat([qk.flatten(1), torch.randn((T, H * V), generator=g, device=DEV)], 1).contiguous()
    beta = torch.sigmoid(torch.randn((T, H), generator=g, device=DEV))
    decay = torch.exp(-torch.rand((T, H), generator=g, device=DEV) * 0.1)
    decay[::13], decay[5::17] = 1.0, 0.0
    state = torch.randn((n + 2, H * D * V + 4), generator=g, device=DEV)
    view, keep = batch(lens, slots)

    def call(s):
        o = torch.zeros((T, H * V), device=DEV)
        scratch = torch.full((B.recurrent_scratch_floats(D, T, H),), float("nan"), device=DEV)
        B.delta_recur(qkv, beta, decay, s, 0, o, G, D, H, V, view, B.stream_ptr(), scratch=scratch)
        return o
    (o, s), (o1, s1) = both_ways(monkeypatch, call, state)
    q, k, v = (x.double() for x in (qkv[:, :G * D].view(T, G, D), qkv[:, G * D:2 * G * D].view(T, G, D), qkv[:, 2 * G * D:].view(T, H, V)))
    q, k = (x.repeat_interleave(H // G, 1) for x in (q, k))
    want_o, want_s, at = torch.zeros((T, H, V), dtype=torch.float64, device=DEV), state.double(), 0
    for i, m in enumerate(lens):
        if slots[i] >= 0:
            S = want_s[slots[i], :H * D * V].view(H, D, V).clone()
            for t in range(at, at + m):
                S = S * decay[t].double()[:, None, None]
                u = beta[t].double()[:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t]))
                S = S + k[t][:, :, None] * u[:, None]
                want_o[t] = torch.einsum("hdv,hd->hv", S, q[t])
            want_s[slots[i], :H * D * V] = S.flatten()
        at += m
    for got, plain, want in ((o, o1, want_o.flatten(1)), (s, s1, want_s)):
        # a sum of up to DIM + 8 terms per token, rounded to 2^-24 each; errors of earlier tokens fade with the decays
        assert off(got, want) <= 2.0 ** -20
        assert off(got, want) <= 1.25 * off(plain, want) + 2.0 ** -25


@pytest.mark.parametrize("D,V,H", [(64, 64, 5), (128, 128, 2), (64, 36, 2), (128, 4, 1)])
@pytest.mark.parametrize("lens", [LENS, [5], [2048], [4] * 8, [31]])
def test_decay_per_key_channel(monkeypatch, D, V, H, lens):
    from inference_engine_rust_b200.csrc import bindings as B
    g = torch.Generator(device=DEV).manual_seed(D + V + len(lens))
    T, n = sum(lens), len(lens)
    slots = list(range(n, 0, -1))
    slots[1 % n] = slots[1 % n] if n == 1 else -1
    x = torch.randn((T, 2 * H * D + H * V + 8), generator=g, device=DEV)
    decay = torch.exp(-torch.exp(torch.rand((T, H * D), generator=g, device=DEV) * 6 - 6))
    decay[::13, ::3], decay[5::17, 1::5] = 1.0, 0.0
    u = torch.randn((H, D), generator=g, device=DEV)
    state = torch.randn((n + 2, H * D * V + 4), generator=g, device=DEV)
    view, keep = batch(lens, slots)

    def call(s):
        o = torch.zeros((T, H * V), device=DEV)
        scratch = torch.full((B.recurrent_scratch_floats(D, T, H),), float("nan"), device=DEV)
        B.wkv_recur(x, decay, u, s, 0, o, D, H, V, view, B.stream_ptr(), scratch=scratch)
        return o
    (o, s), (o1, s1) = both_ways(monkeypatch, call, state)
    r, k, v = (x[:, a:b].double().view(T, H, -1) for a, b in ((0, H * D), (H * D, 2 * H * D), (2 * H * D, 2 * H * D + H * V)))
    w = decay.double().view(T, H, D)
    want_o, want_s, at = torch.zeros((T, H, V), dtype=torch.float64, device=DEV), state.double(), 0
    for i, m in enumerate(lens):
        if slots[i] >= 0:
            S = want_s[slots[i], :H * D * V].view(H, D, V).clone()
            for t in range(at, at + m):
                kv = k[t][:, :, None] * v[t][:, None]
                want_o[t] = torch.einsum("hdv,hd->hv", S + u.double()[:, :, None] * kv, r[t])
                S = S * w[t][:, :, None] + kv
            want_s[slots[i], :H * D * V] = S.flatten()
        at += m
    for got, plain, want in ((o, o1, want_o.flatten(1)), (s, s1, want_s)):
        assert off(got, want) <= 2.0 ** -20
        assert off(got, want) <= 1.25 * off(plain, want) + 2.0 ** -25


@pytest.mark.parametrize("V", [8, 64, 128, 24, 256])
@pytest.mark.parametrize("H,n_tokens", [(3, 1), (5, 7), (64, 300)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_norm_of_the_read_out_and_gate(dtype, H, n_tokens, V):
    """A norm per head, a weight per number (shared by the heads or not) and a gate: at the edges of a block's (token, head)
    pairs, for head sizes that the vector form takes and for others."""
    from inference_engine_rust_b200.csrc import bindings as B
    g = torch.Generator(device=DEV).manual_seed(V + H)
    o = torch.randn((n_tokens, H, V), generator=g, device=DEV)
    proj = (torch.randn((n_tokens, H * V + 16), generator=g, device=DEV) * 3).to(dtype)
    for shared in (True, False):
        w = torch.randn((V if shared else H * V,), generator=g, device=DEV)
        out = torch.empty((n_tokens, H * V), dtype=dtype, device=DEV)
        B.gated_head_norm(o, proj, 16, w, shared, 0 if shared else 1, 1e-5, out, n_tokens, H, V, B.stream_ptr())
        z = proj[:, 16:].double()
        gate = torch.sigmoid(z) * (z if shared else 1.0)
        x = o.double()
        want = (x / torch.sqrt(x.square().mean(-1, keepdim=True) + 1e-5) * (w.double() if shared else w.double().view(H, V))).flatten(1) * gate
        # a few fp32 roundings, and one to the result's type
        assert ((out.double() - want).abs() <= want.abs() * (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -19) + 1e-7).all()


@pytest.mark.parametrize("L,C,width", [(64, 4096, 4096), (12, 516, 100), (4, 4, 7), (24, 1020, 520), (500, 640, 64)])
@pytest.mark.parametrize("lens", [[256], [5, 0, 3, 1, 290, 4, 17], [255 + 1, 1], [1] * 300])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_decays_of_a_prompt(dtype, lens, L, C, width):
    """The product with the decays' matrix, sixteen tokens a block (256 tokens and more), and the rows it keeps: sequences that end
    inside a block, an empty one and one of padding, channels that leave a rest in a block."""
    from inference_engine_rust_b200.csrc import bindings as B
    g = torch.Generator(device=DEV).manual_seed(L + C + len(lens))
    T, n = sum(lens), len(lens)
    slots = list(range(n, 0, -1))
    if n > 1:
        slots[n // 2] = -1
    z = torch.randn((T, L + 4), generator=g, device=DEV) * 2
    w2t = torch.randn((L, C), generator=g, device=DEV) * L ** -0.5
    w0 = torch.rand((C,), generator=g, device=DEV) * 5 - 6
    h = torch.randn((T, width + 3), generator=g, device=DEV).to(dtype)[:, :width]
    state = torch.full((n + 2, width + 9), 7.0, device=DEV)
    decay = torch.full((T + 1, C), 7.0, device=DEV)
    view, keep = batch(lens, slots)
    B.wkv_decay(z, L, w2t, w0, decay, h, state, 5, view, B.stream_ptr())
    torch.cuda.synchronize()
    exponent = torch.exp(w0.double() + torch.tanh(z[:, :L].double()) @ w2t.double())
    want = torch.exp(-exponent)
    # L + 1 rounded additions in the inner exponent (magnitudes of up to |w0| + sum |w2t|), then two exponentials
    off_inner = (L + 4) * 2.0 ** -24 * (w0.double().abs() + w2t.double().abs().sum(0))
    assert ((decay[:T] - want).abs() <= want * (exponent * off_inner * 1.1 + exponent * 2.0 ** -21 + 2.0 ** -21) + 2.0 ** -149).all()
    assert (decay[T] == 7.0).all()
    kept, at = torch.full_like(state, 7.0), 0
    for i, m in enumerate(lens):
        at += m
        if m and slots[i] >= 0:
            kept[slots[i], 5:5 + width] = h[at - 1].float()
    assert torch.equal(state, kept)
