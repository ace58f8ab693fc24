"""Experts' products over the tokens that chose them: the sort of the choices, and the feed-forward against 64-bit arithmetic at
the edges of its row tiles (experts without a token, with one, with a tile and one more), for every router and with portions."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("T,top,E", [(1, 1, 1), (256, 2, 5), (257, 3, 16), (1000, 1, 300), (4096, 2, 16)])
def test_sort(T, top, E):
    from inference_engine_rust_b200.csrc import bindings as B
    g = torch.Generator().manual_seed(T)
    idx = torch.randint(-1, E + 2, (T, top), generator=g, dtype=torch.int32)        # -1 and E, E + 1: no rows
    idx[T // 2:] = E // 2                                                            # one expert takes half of the tokens
    w = torch.rand(T, top, generator=g)
    groups = torch.full((B.moe_group_ints(T, top, E),), -7, dtype=torch.int32, device=DEV)
    pos, row_token = (torch.full((T * top,), -9, dtype=torch.int32, device=DEV) for _ in range(2))
    row_w = torch.zeros(T * top, device=DEV)
    B.moe_sort(idx.to(DEV), w.to(DEV), T, top, E, groups, pos, row_token, row_w, B.stream_ptr())
    groups, pos, row_token, row_w = groups.tolist(), pos.view(T, top).cpu(), row_token.cpu(), row_w.cpu()
    valid = (idx >= 0) & (idx < E)
    assert (pos[~valid] == -1).all() and groups[1] == int(valid.sum())
    assert sorted(pos[valid].tolist()) == list(range(groups[1]))
    t_of = torch.arange(T)[:, None].expand(T, top)
    assert (row_token[pos[valid].long()] == t_of[valid]).all() and (row_w[pos[valid].long()] == w[valid]).all()
    expert_of_row = torch.empty(groups[1], dtype=torch.int32)
    expert_of_row[pos[valid].long()] = idx[valid]
    covered = 0
    for i in range(groups[0]):
        e, first, end = groups[2 + 3 * i:5 + 3 * i]
        last = min(first + 128, end)
        assert first == covered and last > first and (expert_of_row[first:last] == e).all()
        assert end == groups[1] or expert_of_row[end] != e
        covered = last
    assert covered == groups[1]


def part_of(kind, E, top, ff, shared, identity, hidden):
    from inference_engine_rust_b200.config.specs import PartSpec
    from inference_engine_rust_b200.parts import Runtime, part_class
    rt = Runtime(dtype=torch.bfloat16, device=DEV)
    p = {"hidden_size": hidden, "experts": E, "top": top, "expert_ff": ff}
    if kind == "moe":
        p["shared_ff"] = shared
    else:
        p.update(identity=identity, groups=1, keep=1, score="softmax", activation="gelu_tanh")
    part = part_class("ffn", kind)(PartSpec(kind, p), rt)
    g = torch.Generator(device=DEV).manual_seed(E + top)
    w = {n: (torch.randn(s.shape, generator=g, device=DEV) * 0.1).to(torch.bfloat16) for n, s in part.tensor_specs().items()}
    part.load(dict(w))
    return part, w


def exact(kind, part, w, x):
    x = x.double()
    z = x @ w["router"].double().t()
    act = F.silu if kind == "moe" else lambda v: F.gelu(v, approximate="tanh")
    if kind == "moe":
        val, idx = torch.topk(z + w["router.b"].double(), part.top)
        wt = torch.softmax(val, -1)
    else:
        s = torch.softmax(z, -1)
        idx = torch.topk(s + w["correction"].double(), part.top).indices
        wt = torch.gather(s, 1, idx)
        wt = wt / wt.sum(-1, keepdim=True)
    out = torch.zeros_like(x)

    def ff(v, n):
        return (act(v @ w[n + ".gate"].double().t()) * (v @ w[n + ".up"].double().t())) @ w[n + ".down"].double().t()
    for e in range(z.shape[1]):
        t, j = torch.nonzero(idx == e, as_tuple=True)
        if t.numel():
            out[t] += wt[t, j, None] * (ff(x[t], f"e{e}") if e < part.experts else x[t])
    return out + ff(x, "shared") if "shared.gate" in w else out


@pytest.mark.parametrize("kind,E,top,ff,shared,identity", [("moe", 8, 2, 64, 96, 0), ("moe", 40, 3, 192, 0, 0), ("moe", 9, 1, 128, 200, 0),
                                                           ("grouped_moe", 12, 2, 64, 0, 0), ("grouped_moe", 13, 2, 192, 0, 3)])
@pytest.mark.parametrize("T", [256, 385, 1030])
def test_against_64_bits(monkeypatch, kind, E, top, ff, shared, identity, T):
    from inference_engine_rust_b200.parts import StepContext, moe
    part, w = part_of(kind, E, top, ff, shared, identity, 136)
    g = torch.Generator(device=DEV).manual_seed(T)
    x = torch.randn((T, 136), generator=g, device=DEV).to(torch.bfloat16)
    x[: T // 2] = x[0]                                # one choice takes half of the tokens, some take few or none
    ctx = StepContext(kind="prompt", batch=None, n_tokens=T, n_seqs=1, q_lens=[T], pos0=[0], slots=[0],
                      stream=torch.cuda.current_stream().cuda_stream, rt=part.rt)
    base = torch.randn((T, 136), generator=g, device=DEV)
    want = base + exact(kind, part, w, x)
    got = {}
    for name, least, most in (("grouped", 1, 8192), ("portions", 1, 256), ("all experts", 1 << 30, 8192)):
        monkeypatch.setattr(moe, "GROUPED_MIN_TOKENS", least)
        monkeypatch.setattr(moe, "GROUPED_MAX_TOKENS", most)
        assert part._takes_grouped(x, T) == (least == 1)
        got[name] = base.clone()
        part.forward(x, got[name], ctx)
        torch.cuda.synchronize()
        assert part.rt.err.item() == 0
        # bf16 weights and inputs are exact here; an activation is rounded once, by at most 2^-9 of itself
        assert (got[name] - want).norm() <= 2.0 ** -8 * (want - base).norm(), name
    if T % 256 == 0:
        assert torch.equal(got["grouped"], got["portions"])


def test_a_row_that_is_no_number_stays_one():
    from inference_engine_rust_b200.parts import StepContext
    part, w = part_of("moe", 8, 2, 64, 96, 0, 136)
    x = torch.randn((400, 136), device=DEV).to(torch.bfloat16)
    x[7] = float("nan")
    out = torch.zeros((400, 136), device=DEV)
    ctx = StepContext(kind="prompt", batch=None, n_tokens=400, n_seqs=1, q_lens=[400], pos0=[0], slots=[0],
                      stream=torch.cuda.current_stream().cuda_stream, rt=part.rt)
    assert part._takes_grouped(x, 400)
    part.forward(x, out, ctx)
    assert torch.isnan(out[7]).all() and torch.isfinite(out[:7]).all() and torch.isfinite(out[8:]).all()


@pytest.mark.parametrize("T,E,top,K,shared", [(1, 1, 1, 8, False), (3, 5, 2, 264, True), (64, 16, 4, 4096, False), (33, 70, 3, 1000, True)])
def test_router_in_one_kernel(T, E, top, K, shared):
    """The product with the routing behind it, against the two kernels apart on the same 32-bit logits."""
    from inference_engine_rust_b200.csrc import bindings as B
    g = torch.Generator(device=DEV).manual_seed(E)
    x = torch.randn((T, K), generator=g, device=DEV).to(torch.bfloat16)
    w_r = (torch.randn((E, K), generator=g, device=DEV) * K ** -0.5).to(torch.bfloat16)
    bias = torch.randn(E, generator=g, device=DEV) * 0.1
    z = (x.double() @ w_r.double().t()).float()

    def empty():
        return (torch.full((T, E + shared), 9.0, device=DEV), torch.empty((T, top), dtype=torch.int32, device=DEV), torch.empty((T, top), device=DEV))
    for grouped in (None, dict(correction=bias, groups=1, keep=1, score="sigmoid", group_score="top2_sum", weight_scale=2.5)):
        a, b = empty(), empty()
        wid = torch.empty(T, device=DEV)
        if grouped is None:
            assert B.router_step(x, w_r, T, E, top, *a, B.stream_ptr(), bias=bias)
            B.router_topk(z, bias, T, E, top, *b, B.stream_ptr())
        else:
            assert B.router_step(x, w_r, T, E, top, *a, B.stream_ptr(), N=E, wid=wid, grouped=grouped)
            opts = dict(grouped)
            B.router_grouped(z, opts.pop("correction"), T, E, E, top, opts.pop("groups"), opts.pop("keep"), b[0], wid, b[1], b[2], B.stream_ptr(), **opts)
        assert torch.equal(a[1], b[1])
        for p, q in ((a[0], b[0]), (a[2], b[2])):
            assert ((p - q).abs() <= 2.0 ** -16).all()            # logits of size 1 summed in another order, K terms of 2^-24
    assert not B.router_step(x[:, 1:], w_r[:, 1:], T, E, top, *empty(), B.stream_ptr(), bias=bias)


@pytest.mark.parametrize("kind,E,top,ff,shared,identity", [("moe", 8, 2, 64, 96, 0), ("grouped_moe", 13, 2, 192, 0, 3)])
@pytest.mark.parametrize("T", [1, 40, 200, 400])
def test_residual_that_is_a_view(kind, E, top, ff, shared, identity, T):
    """Rows wider than the layer, and rows off the 16-byte boundaries: the same results, and nothing beside them written."""
    from inference_engine_rust_b200.parts import StepContext
    part, w = part_of(kind, E, top, ff, shared, identity, 136)
    g = torch.Generator(device=DEV).manual_seed(T)
    x = torch.randn((T, 136), generator=g, device=DEV).to(torch.bfloat16)
    step = dict(kind="prompt", batch=None, n_tokens=T, n_seqs=1, q_lens=[T], pos0=[0], slots=[0], rt=part.rt)
    base = torch.randn((T, 136), generator=g, device=DEV)
    exactly = exact(kind, part, w, x)
    for width, first in ((136, 0), (160, 0), (160, 8), (139, 0), (160, 1)):
        wide = torch.full((T, width), 5.0, device=DEV)
        res = wide[:, first:first + 136]
        res.copy_(base)
        part.forward(x, res, StepContext(stream=torch.cuda.current_stream().cuda_stream, **step))
        torch.cuda.synchronize()
        assert part.rt.err.item() == 0
        assert (res - base - exactly).norm() <= 2.0 ** -8 * exactly.norm(), (width, first)
        assert (wide[:, :first] == 5.0).all() and (wide[:, first + 136:] == 5.0).all()
    if T == 400:
        assert part._takes_grouped(x, T, base) and part._takes_grouped(x, T, torch.zeros((T, 160), device=DEV)[:, 8:144])
        assert not part._takes_grouped(x, T, torch.zeros((T, 139), device=DEV)[:, :136])
        assert not part._takes_grouped(x, T, torch.zeros((T, 160), device=DEV)[:, 1:137])


@pytest.mark.parametrize("kind,E,top,ff,shared,identity", [("moe", 8, 2, 64, 96, 0), ("grouped_moe", 13, 2, 192, 0, 3)])
@pytest.mark.parametrize("T", [512, 513, 768])
def test_portions(monkeypatch, kind, E, top, ff, shared, identity, T):
    """A prompt in two, three or four portions, bounded by tokens or by bytes: the bits of one portion, and no more workspace than said."""
    from inference_engine_rust_b200.parts import StepContext, Workspace, moe
    part, w = part_of(kind, E, top, ff, shared, identity, 136)
    g = torch.Generator(device=DEV).manual_seed(T)
    x = torch.randn((T, 136), generator=g, device=DEV).to(torch.bfloat16)
    base = torch.randn((T, 136), generator=g, device=DEV)
    a_token = top * (4 * 136 + 2 * ff)
    monkeypatch.setattr(moe, "GROUPED_MIN_TOKENS", 128)
    got = {}
    for most, room, size in ((8192, 1 << 40, T), (256, 1 << 40, 256), (8192, 200 * a_token + 5, 200), (200, 300 * a_token, 200)):
        monkeypatch.setattr(moe, "GROUPED_MAX_TOKENS", most)
        monkeypatch.setattr(moe, "GROUPED_MAX_BYTES", room)
        part.rt.workspace = Workspace(DEV)
        assert part._takes_grouped(x, T) and part._portion() == min(most, room // a_token)
        got[most, room] = base.clone()
        part.forward(x, got[most, room], StepContext(kind="prompt", batch=None, n_tokens=T, n_seqs=1, q_lens=[T], pos0=[0], slots=[0],
                                                     stream=torch.cuda.current_stream().cuda_stream, rt=part.rt))
        torch.cuda.synchronize()
        assert part.rt.err.item() == 0
        per_row = sum(b.numel() for n, b in part.rt.workspace._bufs.items() if n in ("moe.act", "moe.results", "moe.rows"))
        assert per_row <= size * a_token
    first, *others = got.values()
    assert all(torch.equal(first, o) for o in others)
    monkeypatch.setattr(moe, "GROUPED_MAX_BYTES", 127 * a_token)             # portions too small to be worth it
    assert not part._takes_grouped(x, T)


def test_portions_of_one_token():
    """Every kernel of the grouped form at its smallest."""
    part, w = part_of("moe", 8, 2, 64, 96, 0, 136)
    x = torch.randn((5, 136), device=DEV).to(torch.bfloat16)
    out = torch.zeros((5, 136), device=DEV)
    for t in range(5):
        part._forward_grouped(x[t:t + 1], out[t:t + 1], 1, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    want = exact("moe", part, w, x)
    assert part.rt.err.item() == 0 and (out - want).norm() <= 2.0 ** -8 * want.norm()


@pytest.mark.parametrize("kind", ["moe", "grouped_moe"])
@pytest.mark.parametrize("E,one", [(16, True), (17, False), (40, False)])
def test_which_steps_route_in_one_kernel(monkeypatch, kind, E, one):
    from inference_engine_rust_b200.csrc import bindings as B
    from inference_engine_rust_b200.parts import StepContext, moe
    part, w = part_of(kind, E, 2, 64, 0, 0, 136)
    taken = []
    real = B.router_step
    monkeypatch.setattr(B, "router_step", lambda *a, **k: taken.append(real(*a, **k)) or taken[-1])
    for T in (1, 33, 64, 65):
        g = torch.Generator(device=DEV).manual_seed(T)
        x, out = torch.randn((T, 136), generator=g, device=DEV).to(torch.bfloat16), torch.zeros((T, 136), device=DEV)
        taken.clear()
        step = StepContext(kind="decode", batch=None, n_tokens=T, n_seqs=T, q_lens=[1] * T, pos0=[0] * T, slots=list(range(T)),
                           stream=torch.cuda.current_stream().cuda_stream, rt=part.rt)
        part.forward(x, out, step)
        torch.cuda.synchronize()
        assert part.rt.err.item() == 0 and taken == ([True] if one and T <= 64 else [])
        apart = torch.zeros((T, 136), device=DEV)
        with monkeypatch.context() as m:
            m.setattr(moe, "ROUTER_STEP_MAX_TOKENS", 0)
            part.forward(x, apart, step)
        # weights from logits summed in another order (2^-16 at most), behind which an activation may round the other way (2^-8)
        assert (out - apart).norm() <= 2.0 ** -8 * apart.norm()


@pytest.mark.parametrize("E,top,ff,hidden,T,takes", [(48, 6, 256, 1024, 384, True), (48, 7, 256, 1024, 384, False), (48, 6, 256, 1024, 383, False),
                                                     (40, 1, 64, 4096, 767, False), (40, 1, 64, 4096, 768, True),
                                                     (8, 2, 64, 1024, 1024, True), (8, 2, 64, 1024, 1025, False)])
def test_thin_experts_stay_with_all_tokens(E, top, ff, hidden, T, takes):
    from inference_engine_rust_b200.parts import StepContext
    part, w = part_of("moe", E, top, ff, 0, 0, hidden)
    w = {n: t * (136 / hidden) ** 0.5 for n, t in w.items()}
    part.load(dict(w))
    x = torch.randn((T, hidden), generator=torch.Generator(device=DEV).manual_seed(T), device=DEV).to(torch.bfloat16)
    out = torch.zeros((T, hidden), device=DEV)
    assert part._takes_grouped(x, T, out) == takes
    part.forward(x, out, StepContext(kind="prompt", batch=None, n_tokens=T, n_seqs=1, q_lens=[T], pos0=[0], slots=[0],
                                     stream=torch.cuda.current_stream().cuda_stream, rt=part.rt))
    torch.cuda.synchronize()
    want = exact("moe", part, w, x)
    assert part.rt.err.item() == 0 and (out - want).norm() <= 2.0 ** -8 * want.norm()
