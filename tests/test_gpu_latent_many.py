"""One-token latent attention of more than 16 sequences (a head's matrices whole in shared memory in the absorption and in the
merge): against the plain kernels on the same cache, at sizes that leave rests in every tile."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def context(rt, kind, q_lens, pos0, slots):
    from inference_engine_rust_b200.csrc import bindings as B
    from inference_engine_rust_b200.parts import StepContext
    n = len(q_lens)
    arrs = [torch.as_tensor(a, dtype=torch.int32, device=DEV) for a in
            (torch.tensor([0] + q_lens).cumsum(0), slots, torch.arange(n).repeat_interleave(torch.tensor(q_lens)), pos0)]
    view = B.BatchView(cu_q=arrs[0].data_ptr(), slot_ids=arrs[1].data_ptr(), tok_seq=arrs[2].data_ptr(), pos0=arrs[3].data_ptr(),
                       n_seqs=n, n_tokens=sum(q_lens))
    ctx = StepContext(kind=kind, batch=view, n_tokens=sum(q_lens), n_seqs=n, q_lens=list(q_lens), pos0=list(pos0), slots=list(slots),
                      stream=B.stream_ptr(), rt=rt)
    ctx._keep = arrs
    return ctx


@pytest.mark.parametrize("batch", [16, 17, 32, 33, 50])
@pytest.mark.parametrize("heads,dim,rot,vdim,rank,sink", [(5, 36, 16, 40, 64, False), (32, 128, 64, 128, 512, False), (3, 64, 32, 136, 96, False),
                                                          (4, 64, 0, 64, 128, True), (17, 20, 8, 24, 520 - 8, False),
                                                          (64, 16, 8, 24, 40, False), (70, 32, 16, 136, 16, False), (40, 64, 32, 64, 256, False),
                                                          (9, 128, 16, 128, 256, False), (4, 128, 64, 128, 128, False),
                                                          (4, 32, 16, 32, 16, False), (3, 16, 8, 24, 24, False), (20, 32, 0, 32, 32, True),
                                                          (4, 16, 8, 16, 40, False), (33, 64, 16, 136, 56, False)])
def test_against_the_plain_kernels(batch, heads, dim, rot, vdim, rank, sink):
    from inference_engine_rust_b200.cache import Cache
    from inference_engine_rust_b200.config.specs import PartSpec
    from inference_engine_rust_b200.parts import Runtime, part_class
    p = {"hidden_size": 64, "heads": heads, "dim": dim, "vdim": vdim, "kv_rank": rank, "q_rank": 48 if sink else None, "scale": 0.2,
         "eps": 1e-5, "sink": sink}
    if rot:
        p.update(rot_dim=rot, gate="head", position=PartSpec("rope", {"theta": 1e4, "rotary_dim": rot, "pairing": "interleaved"}))
    g = torch.Generator(device=DEV).manual_seed(batch + heads)
    lens = [1 + (37 * i) % 150 for i in range(batch)]
    w = hist = x = None
    out = []
    for plain in (True, False):
        rt = Runtime(dtype=torch.bfloat16, device=DEV, plain_only=plain)
        part = part_class("mixer", "latent_attention")(PartSpec("latent_attention", p), rt)
        if w is None:
            w = {n: (torch.randn(s.shape, generator=g, device=DEV) * 0.3).to(torch.bfloat16) for n, s in part.tensor_specs().items()}
            hist = torch.randn((sum(lens), 64), generator=g, device=DEV).to(torch.bfloat16)
            x = torch.randn((batch, 64), generator=g, device=DEV).to(torch.bfloat16)
        part.load(dict(w))
        cache = Cache({0: part.cache_request()}, max_tokens=64 * 3 * batch, max_seq_len=192, max_sequences=batch, dtype=torch.bfloat16, device=DEV,
                      poison=True)
        slots = [cache.open_sequence() for _ in lens]
        for s, n in zip(slots, lens):
            cache.reserve(s, n + 1)
        cache.upload()
        part.forward(hist, torch.zeros((sum(lens), 64), device=DEV), context(rt, "prompt", lens, [0] * batch, slots), cache.layer_view(0), True)
        padded = list(slots)
        padded[batch // 2] = -1                     # a padding sequence
        res = torch.zeros((batch, 64), device=DEV)
        part.forward(x, res, context(rt, "decode", [1] * batch, lens, padded), cache.layer_view(0), True)
        torch.cuda.synchronize()
        assert rt.err.item() == 0
        keep = [i for i in range(batch) if i != batch // 2]
        out.append(res[keep].double())
    # absorbed queries, probabilities and the heads' results are rounded to bf16 (2^-9 each), in the plain kernels some are not
    assert (out[0] - out[1]).norm() <= 2.0 ** -6 * out[0].norm()
