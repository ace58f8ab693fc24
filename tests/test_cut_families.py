"""A cut by length that mixers of one family ask for reaches the mixers of that family, in every layer and on both sides of a pair, and no others."""
from types import SimpleNamespace

import pytest


class Toy:
    def __init__(self, family, longest):
        self.cut_family, self.longest, self.seen = family, longest, []

    def cut_by_length_key(self):
        return (self.cut_family, self.longest)

    def cut_by_length(self, pos0, cache_view):
        assert cache_view == "view"
        return max(pos0) > self.longest

    def forward(self, xn, residual, ctx, cache_view, writes_cache):
        self.seen.append(ctx.unequal_lengths)


class Silent:                                        # a mixer of a user's own, without the question
    def __init__(self):
        self.seen = []

    def forward(self, xn, residual, ctx, cache_view, writes_cache):
        self.seen.append(ctx.unequal_lengths)


def layers_of(monkeypatch, mixers):
    """A model of these mixers that launches nothing."""
    from inference_engine_rust_b200.engine import model as M
    monkeypatch.setattr(M.B, "embed_gather", lambda *a, **k: None)
    model = M.Model.__new__(M.Model)
    block = lambda m: SimpleNamespace(forward=lambda rows, ctx, view, writes: m.forward(rows, rows, ctx, view, writes))
    model.spec = SimpleNamespace(hidden_size=8, schedule=[SimpleNamespace(layer=i, pass_start=None, writes_cache=True) for i in range(len(mixers))],
                                 cache_entry=lambda pos: pos, residual_streams=None, embedding_scale=1.0)
    model.rt = SimpleNamespace(workspace=SimpleNamespace(take=lambda *a: None), err=None)
    model._layer_parts = [(None, m, None, None) for m in mixers]
    model.blocks = [block(m) for m in mixers]
    model.inputs, model.passes, model.after_block, model.embedding, model._cut_askers = [], None, None, None, None
    return model


@pytest.mark.parametrize("longest,want", [(50, set()), (150, {"latent"}), (250, {"latent", "attention"})])
def test_a_family_gets_its_own_answer(monkeypatch, longest, want):
    from inference_engine_rust_b200.parts import StepContext
    from inference_engine_rust_b200.parts.parallel import ParallelMixers
    pair = ParallelMixers.__new__(ParallelMixers)
    pair.subs = [Toy("latent", 100), Toy("attention", 200)]
    latent, attention, other, silent = Toy("latent", 100), Toy("attention", 200), Toy("attention", 1000), Silent()
    model = layers_of(monkeypatch, [latent, attention, pair, other, silent])
    views = {2: ("view", "view")}
    cache = SimpleNamespace(layer_view=lambda entry: views.get(entry, "view"))
    families = model.cut_by_length([3, longest, 7], cache)
    assert set(families) == want
    ctx = StepContext(kind="decode", batch=None, n_tokens=3, n_seqs=3, q_lens=[1] * 3, pos0=[3, longest, 7], slots=[0, 1, 2], stream=0, rt=model.rt)
    ctx.cut_families = families
    model.forward(ctx, None, cache, None, 0)
    for mixer in (latent, attention, other, *pair.subs):
        assert mixer.seen == [mixer.cut_family in want]
    assert silent.seen == ["attention" in want]


def test_families_of_the_parts():
    from inference_engine_rust_b200.parts import part_class
    assert part_class("mixer", "latent_attention").cut_family == "latent"
    assert {part_class("mixer", kind).cut_family for kind in ("attention", "gated_attention", "tied_kv_attention")} == {"attention"}
