"""When latent attention asks for a cut by length: what the kernel does, launched for as many sequences as the step is padded to, where that saves enough."""
import random
from types import SimpleNamespace

import pytest
import torch

SMS = 148


def plan(n_seqs, H, rank, rot, width):
    """The launch's plan on 148 SMs (16 heads a tile, 32 where there are more): as many runs as end soonest."""
    hpad = 16 if H <= 16 else -(-H // 32) * 32
    ctas = n_seqs * (1 if H <= 16 else hpad // 32)
    return hpad, min(range(1, 33), key=lambda k: (-(-ctas * k // SMS) * (-(-width // k) + 2), k))


def part_of(monkeypatch, heads, window=None):
    from inference_engine_rust_b200.parts import latent_attention as L
    monkeypatch.setattr(L.B, "latent_decode_tc_plan", plan)
    monkeypatch.setattr(L.B, "latent_decode_tc_rows", lambda n, H, rank, rot, splits: splits + 4 if n >= 8 and splits <= 8 else splits)
    monkeypatch.setattr(L.B, "sm_count", lambda: SMS)
    part = L.LatentAttention.__new__(L.LatentAttention)
    part.rt = SimpleNamespace(fast=True, dtype=torch.bfloat16)
    part.H, part.kv_rank, part.R, part.window, part.plain_form = heads, 512, 64, window, False
    return part


VIEW = SimpleNamespace(group=SimpleNamespace(page_tokens=64, table_width=64, ring_pages=64))


def test_asked_for_the_padded_batch(monkeypatch):
    part = part_of(monkeypatch, 32)
    lens = [4000] + [500] * 79
    assert plan(80, 32, 512, 64, 64)[1] == 5 and plan(128, 32, 512, 64, 64)[1] == 1
    assert not part.cut_by_length(lens, VIEW)                     # (five runs each: the longest is short enough)
    assert part.cut_by_length(lens, VIEW, 128)                    # one CTA for 63 pages
    # the model passes the number on to mixers that want it, beside others that take two arguments
    from inference_engine_rust_b200.engine.model import Model
    model = Model.__new__(Model)
    other = SimpleNamespace(cut_by_length=lambda pos0, view: len(pos0) == 3)
    model.spec = SimpleNamespace(schedule=[SimpleNamespace(layer=0), SimpleNamespace(layer=1)], cache_entry=lambda pos: pos)
    model._layer_parts, model._cut_askers = [(None, part, None, None), (None, other, None, None)], None
    cache = SimpleNamespace(layer_view=lambda entry: VIEW)
    assert model.cut_by_length(lens, cache, 128) == {"latent"} and not model.cut_by_length(lens, cache, 80)
    assert not model.cut_by_length(lens, cache) and model.cut_by_length([1, 2, 3], cache, 4) == {"attention"}


@pytest.mark.parametrize("heads,ctas", [(16, 148), (32, 148), (64, 74), (100, 37)])
@pytest.mark.parametrize("window", [None, 200])
def test_as_the_kernel_cuts(monkeypatch, heads, ctas, window):
    """Against the definition: the fewest pages a run with which all runs have a CTA at once and a sequence's partial results have room,
    where an even run is over three times a CTA's share and longer than that, by four pages at least."""
    part, rng, cut = part_of(monkeypatch, heads, window), random.Random(heads), 0
    for _ in range(400):
        n = rng.randint(1, 160)
        n_seqs = rng.choice([n, 1 << (n - 1).bit_length()])
        low, high = sorted(rng.randint(0, 4095) for _ in range(2))
        lens = [rng.randint(low, high) if rng.random() < 0.1 else rng.randint(0, low) for _ in range(n)]
        splits = plan(n_seqs, heads, 512, 64, 64)[1]
        rows = splits + 4 if n_seqs >= 8 and splits <= 8 else splits
        pages = [p // 64 + 1 - (max(0, p + 1 - window) // 64 if window else 0) for p in lens]
        even = -(-max(pages) // splits)
        fits = [r for r in range(1, 65) if all(-(-x // r) <= rows for x in pages) and sum(-(-x // r) for x in pages) <= ctas]
        want = rows > splits and even * ctas > 3 * sum(pages) and bool(fits) and fits[0] <= even - 4
        assert part.cut_by_length(lens, VIEW, n_seqs) == want, (lens, n_seqs)
        cut += want
    assert window or 20 < cut < 380
