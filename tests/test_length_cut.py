"""When a one-token step's attention is cut by the sequences' lengths: batches of either kind for which both were measured (32 heads over 8
of 128, pages of 64, 296 slots)."""
import pytest


@pytest.mark.parametrize("lengths,cut", [
    ([300] * 64, False), ([2100] * 64, False), ([1000] * 48, False), ([1000] * 128, False), ([4000] * 128, False),                                   # equal
    ([1500] * 4 + [500] * 44, False), ([1500] * 4 + [500] * 124, False), ([3000] * 2 + [200] * 126, False),         # not worth it
    ([3000] * 2 + [200] * 22, True), ([8000] + [200] * 63, True), ([8000] + [200] * 127, True), ([8000] + [200] * 23, True),
    ([2047] * 49, True), ([2100] * 40, True), ([4096] * 20, False),                                     # a last round mostly empty
    # a batch that leaves room: by the average alone
    ([1000] * 8, False), ([1500, 500, 500, 500], True), ([900, 800, 700], False)])
def test_wants_length_cut(monkeypatch, lengths, cut):
    from inference_engine_rust_b200.parts import fast_attention
    monkeypatch.setattr(fast_attention, "_slots", lambda head_dim: 296)
    assert fast_attention.wants_length_cut(lengths, 8, 4, None, 64, 128) == cut
    assert not fast_attention.wants_length_cut(lengths[:1], 8, 4, None, 64, 128)
