"""The recurrence with a decay per key channel where a launch has more blocks than the device has SMs, and its mixer where a prompt's four
projections are one launch."""
import pytest
import torch

from test_gpu_latent_many import DEV, context
from test_gpu_recurrent_chunks import batch, both_ways, off

pytestmark = pytest.mark.gpu


def test_many_blocks(monkeypatch):
    """Three prompts of 64 heads are 384 blocks, two an SM; one of them alone has an SM for each block and the same bits."""
    from inference_engine_rust_b200.csrc import bindings as B
    D = V = 64
    H, lens = 64, [50, 61, 48]
    assert 2 * H * len(lens) > 2 * B.sm_count() >= 2 * H
    T, g = sum(lens), torch.Generator(device=DEV).manual_seed(3)
    x = torch.randn((T, 3 * H * D), generator=g, device=DEV)
    decay = torch.exp(-torch.exp(torch.rand((T, H * D), generator=g, device=DEV) * 6 - 6))
    u = torch.randn((H, D), generator=g, device=DEV)
    state = torch.randn((3, H * D * V), generator=g, device=DEV)

    def run(lens, first):
        view, keep = batch(lens, list(range(len(lens))))
        n = sum(lens)

        def call(s, keep=keep):                        # (the launch reads the arrays behind the view)
            o = torch.zeros((n, H * V), device=DEV)
            scratch = torch.full((B.recurrent_scratch_floats(D, n, H),), float("nan"), device=DEV)
            B.wkv_recur(x[first:first + n], decay[first:first + n], u, s, 0, o, D, H, V, view, B.stream_ptr(), scratch=scratch)
            return o
        return call
    (o, s), (o1, s1) = both_ways(monkeypatch, run(lens, 0), state)
    r, k, v = (x[:, i * H * D:(i + 1) * H * D].double().view(T, H, -1) for i in range(3))
    w = decay.double().view(T, H, D)
    want_o, want_s, at = torch.zeros((T, H, V), dtype=torch.float64, device=DEV), state.double().view(3, H, D, V).clone(), 0
    for i, m in enumerate(lens):
        for t in range(at, at + m):
            kv = k[t][:, :, None] * v[t][:, None]
            want_o[t] = torch.einsum("hdv,hd->hv", want_s[i] + u.double()[:, :, None] * kv, r[t])
            want_s[i] = want_s[i] * w[t][:, :, None] + kv
        alone = state[i:i + 1].clone()
        assert torch.equal(run([m], at)(alone), o[at:at + m]) and torch.equal(alone[0], s[i])
        at += m
    for got, plain, want in ((o, o1, want_o.flatten(1)), (s, s1, want_s.flatten(1))):
        # sums of up to DIM + 16 terms, rounded to 2^-24 each, as in the kernel that goes token after token
        assert off(got, want) <= 2.0 ** -20
        assert off(got, want) <= 1.25 * off(plain, want) + 2.0 ** -25


@pytest.mark.parametrize("lens", [[65, 100], [48], [47, 17], [33, 1, 0, 9]])       # (sixteen tokens at a time, and eight)
def test_scratch_is_as_large_as_asked_for(lens):
    from inference_engine_rust_b200.csrc import bindings as B
    D = V = 64
    H, T, g = 3, sum(lens), torch.Generator(device=DEV).manual_seed(len(lens))
    x = torch.randn((T, 3 * H * D), generator=g, device=DEV)
    decay = torch.exp(-torch.exp(torch.rand((T, H * D), generator=g, device=DEV) * 6 - 6))
    u = torch.randn((H, D), generator=g, device=DEV)
    state = torch.randn((len(lens), H * D * V), generator=g, device=DEV)
    view, keep = batch(lens, list(range(len(lens))))
    n, res = B.wkv_scratch_floats(D, T, H), []
    assert n == 16 * T * H <= B.recurrent_scratch_floats(D, T, H)
    for room in (n, B.recurrent_scratch_floats(D, T, H)):
        scratch = torch.full((room + 4096,), 7.0, device=DEV)       # (room behind it, so that a write too far is seen and harms nothing)
        s, o = state.clone(), torch.zeros((T, H * V), device=DEV)
        B.wkv_recur(x, decay, u, s, 0, o, D, H, V, view, B.stream_ptr(), scratch=scratch)
        torch.cuda.synchronize()
        assert (scratch[n:] == 7.0).all()
        res.append((o, s))
    assert torch.equal(res[0][0], res[1][0]) and torch.equal(res[0][1], res[1][1])


@pytest.mark.parametrize("lens,together", [([300], True), ([200, 57], True), ([256], False)])
def test_four_projections_in_one_launch(monkeypatch, lens, together):
    from inference_engine_rust_b200.cache import Cache
    from inference_engine_rust_b200.config.specs import PartSpec
    from inference_engine_rust_b200.csrc import bindings as B
    from inference_engine_rust_b200.parts import Runtime, part_class
    p = {"hidden_size": 72, "heads": 4, "dim": 64, "decay_rank": 16, "eps": 1e-5}
    g = torch.Generator(device=DEV).manual_seed(sum(lens))
    said, ask = [], B.gemm_tc_batched

    def asked(*a):
        said.append(ask(*a))
        return said[-1]
    w = xn = None
    res = []
    for way in ("one launch", "one by one", "plain kernels"):
        monkeypatch.setattr(B, "gemm_tc_batched", asked if way == "one launch" else lambda *a: False)
        rt = Runtime(dtype=torch.bfloat16, device=torch.device(DEV), plain_only=way == "plain kernels")
        part = part_class("mixer", "wkv")(PartSpec("wkv", p), rt)
        if w is None:
            w = {n: torch.randn(s.shape, generator=g, device=DEV) * 0.1 for n, s in part.tensor_specs().items()}
            xn = torch.randn((sum(lens), 72), generator=g, device=DEV).bfloat16()
        part.load(dict(w))
        cache = Cache({0: part.cache_request()}, max_tokens=64, max_seq_len=64, max_sequences=len(lens), dtype=torch.bfloat16, device=DEV)
        slots = [cache.open_sequence() for _ in lens]
        out = torch.zeros((sum(lens), 72), device=DEV)
        part.forward(xn, out, context(rt, "prompt", lens, [0] * len(lens), slots), cache.layer_view(0), True)
        torch.cuda.synchronize()
        assert rt.err.item() == 0
        res.append((out.double(), cache.layer_view(0).state[slots].double()))
    assert said == ([True] if together else [])
    (out, state), (out1, state1), (out2, state2) = res
    # the four products are the same sums of 72 bfloat16 products in fp32, whatever kernel adds them; the state holds k and v of all tokens
    assert (state - state1).norm() <= 2.0 ** -20 * state1.norm() and (state - state2).norm() <= 2.0 ** -16 * state2.norm()
    # the read-out is rounded to bfloat16 (2^-9) in front of the last product
    assert (out - out1).norm() <= 2.0 ** -8 * out1.norm() and (out - out2).norm() <= 2.0 ** -8 * out2.norm()
