"""The recurrences over prompts, sixteen tokens at a time, where numbers come near the largest of fp32, which bf16 rounds to infinity, and
where they are infinite: as the kernels that go token after token."""
import pytest
import torch

from test_gpu_recurrent_chunks import DEV, batch, both_ways
from test_gpu_recurrent_sixteen import delta_call, delta_inputs

pytestmark = pytest.mark.gpu
MOST = torch.finfo(torch.float32).max                 # 3.4028e38; bf16's largest is 3.3895e38


def close(got, plain, axis):
    """Column by column; sums of DIM + 16 products rounded to 2^-24 each, in another order."""
    assert torch.isfinite(got).all() and torch.isfinite(plain).all()
    a, b = got.double(), plain.double()
    assert ((a - b).norm(dim=axis) <= 2.0 ** -18 * b.norm(dim=axis)).all()


@pytest.mark.parametrize("D,V", [(128, 128), (64, 44)])
@pytest.mark.parametrize("where", ["value", "state"])
def test_delta_rule_near_the_largest_number(monkeypatch, D, V, where):
    G, H, lens = 1, 2, [48, 32]
    qkv, beta, decay, g = delta_inputs(80, G, D, H, V, D)
    state = torch.randn((2, H * D * V), generator=g, device=DEV)
    if where == "value":
        beta[21, 1] = 1.0
        qkv[21, 2 * G * D + V + 37] = -MOST                        # head 1, column 37
    else:
        state.view(2, H, D, V)[0, 1, 5, 37] = MOST
    view, keep = batch(lens, [0, 1])
    (o, s), (o1, s1) = both_ways(monkeypatch, delta_call(qkv, beta, decay, G, D, H, V, view), state)
    close(o.view(80, H, V)[:48], o1.view(80, H, V)[:48], 0)
    close(o.view(80, H, V)[48:], o1.view(80, H, V)[48:], 0)
    close(s.view(2, H, D, V), s1.view(2, H, D, V), 2)


def wkv(x, decay, u, H, V, view):
    from inference_engine_rust_b200.csrc import bindings as B
    T = x.shape[0]

    def call(s):
        o = torch.zeros((T, H * V), device=DEV)
        scratch = torch.full((B.recurrent_scratch_floats(64, T, H),), float("nan"), device=DEV)
        B.wkv_recur(x, decay, u, s, 0, o, 64, H, V, view, B.stream_ptr(), scratch=scratch)
        return o
    return call


@pytest.mark.parametrize("where,number", [("value", MOST), ("value", -MOST), ("key", MOST), ("state", -MOST), ("value", float("inf")),
                                          ("value", float("-inf")), ("state", float("inf")), ("key", float("inf"))])
def test_decay_per_key_channel_near_the_largest_number(monkeypatch, where, number):
    D, V, H, lens = 64, 44, 3, [63, 80]
    T, g = sum(lens), torch.Generator(device=DEV).manual_seed(7)
    # (small enough that no sum leaves fp32)
    x = torch.randn((T, 2 * H * D + H * V), generator=g, device=DEV) * 2.0 ** -6
    decay = torch.exp(-torch.exp(torch.rand((T, H * D), generator=g, device=DEV) * 6 - 6))
    u = torch.rand((H, D), generator=g, device=DEV) - 0.5
    state = torch.randn((2, H * D * V), generator=g, device=DEV)
    if where == "state":
        state.view(2, H, D, V)[0, 1, 5, 37] = number
    else:
        x[20, (2 * H * D + V + 37) if where == "value" else (H * D + D + 37)] = number          # head 1, column or row 37
    view, keep = batch(lens, [0, 1])
    (o, s), (o1, s1) = both_ways(monkeypatch, wkv(x, decay, u, H, V, view), state)
    if abs(number) <= MOST:
        for at in (slice(0, 63), slice(63, T)):
            close(o.view(T, H, V)[at], o1.view(T, H, V)[at], 0)
        close(s.view(2, H, D, V), s1.view(2, H, D, V), 2)
    else:
        assert torch.equal(torch.isfinite(o), torch.isfinite(o1))
        assert torch.equal(torch.isnan(s), torch.isnan(s1)) and not torch.isnan(s).any()
        assert torch.equal(s == float("inf"), s1 == float("inf")) and torch.equal(s == float("-inf"), s1 == float("-inf"))
