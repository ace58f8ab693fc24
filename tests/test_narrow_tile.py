"""Token tiles of products with few outputs: on both sides of every line of the rule, on 148 SMs."""
from types import SimpleNamespace

import pytest


@pytest.mark.parametrize("outputs,rows,tile", [
    (64, 128, 0), (64, 129, 64), (128, 256, 64), (64, 257, 64), (64, 49 * 64, 64), (64, 49 * 64 + 1, 256),
    (129, 129, 0), (288, 169, 0), (288, 256, 0), (288, 257, 64), (288, 16 * 64, 64), (288, 16 * 64 + 1, 256), (288, 4096, 256), (288, 40, 0)])
def test_narrow_tile(monkeypatch, outputs, rows, tile):
    from inference_engine_rust_b200.parts import fast_linear
    monkeypatch.setattr(fast_linear.B, "sm_count", lambda: 148)
    assert fast_linear.narrow_tile(SimpleNamespace(narrow=True, out_features=outputs), rows) == tile
    assert fast_linear.narrow_tile(SimpleNamespace(narrow=False, out_features=outputs), rows) == 0
