"""One-token latent attention cut by the sequences' lengths: the same results as with every sequence cut into as many runs as the others."""
import pytest
import torch

from test_gpu_latent_many import DEV, context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens", [[1500] + [3, 63, 64, 65, 127, 128, 1] * 2, [700, 2, 650, 5, 610, 300, 64, 1], [2000] + [40] * 70, [100, 260] * 75])
@pytest.mark.parametrize("heads,rank", [(32, 512), (5, 64), (40, 128)])
def test_cut_by_length(lens, heads, rank):
    from inference_engine_rust_b200.cache import Cache
    from inference_engine_rust_b200.config.specs import PartSpec
    from inference_engine_rust_b200.csrc import bindings as B
    from inference_engine_rust_b200.parts import Runtime, part_class
    p = {"hidden_size": 64, "heads": heads, "dim": 32, "vdim": 32, "kv_rank": rank, "q_rank": None, "scale": 0.2, "eps": 1e-5, "sink": False,
         "rot_dim": 16, "gate": "head", "position": PartSpec("rope", {"theta": 1e4, "rotary_dim": 16, "pairing": "interleaved"})}
    g = torch.Generator(device=DEV).manual_seed(len(lens) + heads)
    batch, rt = len(lens), Runtime(dtype=torch.bfloat16, device=DEV)
    part = part_class("mixer", "latent_attention")(PartSpec("latent_attention", p), rt)
    part.load({n: (torch.randn(s.shape, generator=g, device=DEV) * 0.3).to(torch.bfloat16) for n, s in part.tensor_specs().items()})
    pages = sum(n // 64 + 1 for n in lens)
    cache = Cache({0: part.cache_request()}, max_tokens=64 * pages, max_seq_len=64 * (max(lens) // 64 + 1), max_sequences=batch,
                  dtype=torch.bfloat16, device=DEV, poison=True)
    slots = [cache.open_sequence() for _ in lens]
    for s, n in zip(slots, lens):
        cache.reserve(s, n + 1)
    cache.upload()
    hist = torch.randn((sum(lens), 64), generator=g, device=DEV).to(torch.bfloat16)
    part.forward(hist, torch.zeros((sum(lens), 64), device=DEV), context(rt, "prompt", lens, [0] * batch, slots), cache.layer_view(0), True)
    x = torch.randn((batch, 64), generator=g, device=DEV).to(torch.bfloat16)
    padded = list(slots)
    padded[2] = -1
    out = []
    for by_length in (True, False):
        ctx = context(rt, "decode", [1] * batch, lens, padded)
        ctx.unequal_lengths = by_length
        if batch == 71:                              # two runs a sequence; one of 32 pages among seventy of one
            assert part.cut_by_length(lens, cache.layer_view(0)) and not part.cut_by_length([900] * batch, cache.layer_view(0))
        res = torch.zeros((batch, 64), device=DEV)
        part.forward(x, res, ctx, cache.layer_view(0), True)
        torch.cuda.synchronize()
        assert rt.err.item() == 0
        out.append(res[[i for i in range(batch) if i != 2]].double())
    # probabilities are rounded to bf16 (2^-9) against another reference maximum per run
    assert torch.isfinite(out[0]).all()
    assert (out[0] - out[1]).norm() <= 2.0 ** -8 * out[1].norm()


@pytest.mark.parametrize("heads,rank,lens,cut", [
    (32, 512, [4000] + [300] * 63, True), (5, 64, [2000, 1900] + [20] * 30, True), (40, 128, [3000] + [100] * 40, True),
    (32, 64, [700] * 3 + [4050] + [1, 64, 128, 63] * 20, True),
    (40, 128, [4000] + [10] * 99, False),                      # worth it, but more sequences than CTAs
    (32, 64, [500] * 20, False)])                              # not worth it: room for more runs, of which none is used
def test_launches_with_room_for_a_cut(heads, rank, lens, cut):
    """The kernel that works out the cut, over partial results that hold NaN where nobody writes: those a cut takes, those it leaves, and all
    beside the even runs where it takes none."""
    from inference_engine_rust_b200.cache import Cache
    from inference_engine_rust_b200.config.specs import PartSpec
    from inference_engine_rust_b200.csrc import bindings as B
    from inference_engine_rust_b200.parts import Runtime, part_class
    p = {"hidden_size": 64, "heads": heads, "dim": 32, "vdim": 32, "kv_rank": rank, "q_rank": None, "scale": 0.2, "eps": 1e-5, "sink": False,
         "rot_dim": 16, "gate": "head", "position": PartSpec("rope", {"theta": 1e4, "rotary_dim": 16, "pairing": "interleaved"})}
    g = torch.Generator(device=DEV).manual_seed(len(lens) + heads)
    batch, rt = len(lens), Runtime(dtype=torch.bfloat16, device=DEV)
    part = part_class("mixer", "latent_attention")(PartSpec("latent_attention", p), rt)
    part.load({n: (torch.randn(s.shape, generator=g, device=DEV) * 0.3).to(torch.bfloat16) for n, s in part.tensor_specs().items()})
    pages = [n // 64 + 1 for n in lens]
    cache = Cache({0: part.cache_request()}, max_tokens=64 * sum(pages), max_seq_len=64 * max(pages), max_sequences=batch, dtype=torch.bfloat16,
                  device=DEV, poison=True)
    slots = [cache.open_sequence() for _ in lens]
    for s, n in zip(slots, lens):
        cache.reserve(s, n + 1)
    cache.upload()
    hist = torch.randn((sum(lens), 64), generator=g, device=DEV).to(torch.bfloat16)
    part.forward(hist, torch.zeros((sum(lens), 64), device=DEV), context(rt, "prompt", lens, [0] * batch, slots), cache.layer_view(0), True)
    x = torch.randn((batch, 64), generator=g, device=DEV).to(torch.bfloat16)
    hpad, splits = B.latent_decode_tc_plan(batch, heads, rank, 16, max(pages))
    rows = B.latent_decode_tc_rows(batch, heads, rank, 16, splits)
    assert rows > splits
    # the kernel's rule: the fewest pages a run with which every run has a CTA and a partial result, if an even run is longer
    ctas, even = B.sm_count() // (hpad // (32 if heads > 16 else 16)), -(-max(pages) // splits)
    fits = [r for r in range(1, max(pages) + 1) if max(pages) <= r * rows and sum(-(-n // r) for n in pages) <= ctas]
    assert (even * ctas > 3 * sum(pages) and bool(fits) and fits[0] < even) == cut
    assert part.cut_by_length(lens, cache.layer_view(0)) == cut
    out = []
    for by_length in (True, False):
        for name, shape in (("m", (hpad,)), ("l", (hpad,)), ("acc", (hpad, rank))):
            rt.workspace.take("latent.part_" + name, (batch, rows) + shape, torch.float32).fill_(float("nan"))
        ctx = context(rt, "decode", [1] * batch, lens, slots)
        ctx.unequal_lengths = by_length
        res = torch.zeros((batch, 64), device=DEV)
        part.forward(x, res, ctx, cache.layer_view(0), True)
        torch.cuda.synchronize()
        assert rt.err.item() == 0
        out.append(res.double())
    # probabilities are rounded to bf16 (2^-9) against another reference maximum per run
    assert torch.isfinite(out[0]).all()
    assert (out[0] - out[1]).norm() <= 2.0 ** -8 * out[1].norm()
    if not cut:
        assert torch.equal(out[0], out[1])                     # the same even runs
