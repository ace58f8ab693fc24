"""The fp32 projection on the tensor cores (three bf16 parts per number) at the edges of its tiles, blocks and splits, against
64-bit products; what it refuses; infinities and NaN."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def run(x, w, out, M, mode=0):
    from inference_engine_rust_b200.csrc import bindings as B
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    done = B.gemm_f32_tc(x, w, out, M, mode, err, B.stream_ptr())
    torch.cuda.synchronize()
    assert err.item() == 0
    return done


@pytest.mark.parametrize("N,K", [(136, 1024), (130, 1028), (4100, 1056), (2300, 1100), (9300, 1024), (1, 4096)])
@pytest.mark.parametrize("M", [1, 16, 17, 33, 64, 65, 129, 300])
def test_against_64_bits(M, N, K):
    torch.manual_seed(M + N)
    x, w = torch.randn(M, K + 4, device=DEV)[:, :K], torch.randn(N, K, device=DEV)      # (rows with a stride of their own)
    x[0] *= 1e-6
    out = torch.full((M, N + 3), 5.0, device=DEV)
    assert run(x, w, out[:, :N], M)
    ref = x.double() @ w.double().t()
    # K / 64 rounded additions and twelve truncating ones per 64 k, each at most 2^-23 of the sum of magnitudes it meets
    bound = 2.0 ** -19 * (x.double().abs() @ w.double().abs().t())
    assert ((out[:, :N] - ref).abs() <= bound).all()
    assert ((out[:, :N] - ref).norm() <= 2.0 ** -21 * ref.norm())                        # (as random signs add up)
    assert (out[:, N:] == 5.0).all()
    res = torch.randn(M, N, device=DEV)
    total = res.clone()
    assert run(x, w, total, M, mode=1)
    assert torch.equal(total, res + out[:, :N])
    # a row's result does not depend on how many rows the call has
    one = torch.empty(1, N, device=DEV)
    assert run(x[M - 1:], w, one, 1)
    assert torch.equal(one[0], out[M - 1, :N])


def test_refusals():
    x, w, out = torch.randn(4, 1026, device=DEV), torch.randn(8, 1026, device=DEV), torch.empty(4, 8, device=DEV)
    assert not run(x, w, out, 4)                                     # K no multiple of 4
    assert not run(x[:, :1000].contiguous(), w[:, :1000].contiguous(), out, 4)          # short sums: the plain kernel's
    assert not run(x[:, 1:1025], w[:, 1:1025], out, 4)               # rows off the 16-byte boundaries
    assert not run(x.bfloat16(), w.bfloat16(), out, 4)


def test_infinities_and_nan():
    from inference_engine_rust_b200.csrc import bindings as B
    torch.manual_seed(5)
    x, w = torch.randn(40, 1024, device=DEV), torch.randn(300, 1024, device=DEV)
    x[3, 7], x[5, 9], w[11, 70], w[12] = float("inf"), float("nan"), float("-inf"), 0.0
    x[9] *= 1e30
    w[100] *= 1e20
    a, b = torch.empty(40, 300, device=DEV), torch.empty(40, 300, device=DEV)
    B.gemm_plain(x, w, a, 40, 0, B.stream_ptr())
    assert run(x, w, b, 40)
    for same in (torch.isnan, torch.isposinf, torch.isneginf):
        assert torch.equal(same(a), same(b))
    fine = torch.isfinite(a)
    assert ((a - b)[fine].abs() <= 1e-4 * a[fine].abs().max()).all()


@pytest.mark.parametrize("K", [1024, 4100])
@pytest.mark.parametrize("kind", ["one number", "eight numbers", "one large number", "positive", "cut remainders", "rounded remainders"])
def test_error_beside_the_plain_kernel(kind, K):
    """Sums in which one product counts, or all have one sign: no further from 64 bits than one fp32 sum is."""
    from inference_engine_rust_b200.csrc import bindings as B
    torch.manual_seed(K)
    M, N = 40, 300
    x, w = torch.randn(M, K, device=DEV), torch.randn(N, K, device=DEV)
    # mantissas that parts cut off instead of rounded would serve worst
    odd = torch.tensor([0x3f80ffff, 0x3f807fff, 0x3f8080ff, 0x3f817f7f], dtype=torch.int32, device=DEV).view(torch.float32)
    if kind.endswith("numbers") or kind == "one number":
        n = 1 if kind == "one number" else 8
        keep = torch.zeros(M, K, device=DEV).scatter_(1, torch.rand(M, K, device=DEV).topk(n, dim=1).indices, 1.0)
        x = x * keep
        w[::2] = odd[torch.randint(0, 4, (N // 2, K), device=DEV)]
        x[::2] = keep[::2] * odd[torch.randint(0, 4, (M // 2, K), device=DEV)]
    elif kind == "one large number":
        x *= 1e-4
        x[:, 17] = 50.0 + torch.randn(M, device=DEV)
    elif kind == "positive":
        x, w = x.abs(), w.abs()
    elif kind == "cut remainders":
        x, w = odd[torch.randint(0, 4, (M, K), device=DEV)], odd[torch.randint(0, 4, (N, K), device=DEV)]
    else:            # the largest remainders after rounding: 1 + 2^-8 - 2^-16 + 2^-17 - 2^-23, alone in its row
        x, w = torch.zeros(M, K, device=DEV), torch.full((N, K), 0x3f807f3f, dtype=torch.int32, device=DEV).view(torch.float32)
        x[:, 70] = w[0, 0]
    tc, plain = torch.empty(M, N, device=DEV), torch.empty(M, N, device=DEV)
    assert run(x, w, tc, M)
    B.gemm_plain(x, w, plain, M, 0, B.stream_ptr())
    ref = x.double() @ w.double().t()
    off, beside = (tc - ref).norm(), (plain - ref).norm()
    # one product: a rounding of 2^-24 in both kernels, and here the products left out: 2^-24 at most, mostly far less
    assert off <= (beside + 2.0 ** -24 * ref.norm() if kind == "rounded remainders" else 1.1 * beside)
    if kind in ("one number", "rounded remainders"):
        assert ((tc - ref).abs() <= 2.0 ** -23 * ref.abs()).all()


@pytest.mark.parametrize("exponent", [-40, -58, -80, -100, -112, -122])
@pytest.mark.parametrize("M,N", [(1, 140), (40, 300), (130, 9300)])
def test_small_numbers(exponent, M, N):
    """Rows whose numbers lose bits below bf16's smallest number: what comes out is as precise as the plain kernel's."""
    from inference_engine_rust_b200.csrc import bindings as B
    torch.manual_seed(M)
    x, w = torch.randn(M, 1024, device=DEV) * 2.0 ** exponent, torch.randn(N, 1024, device=DEV)
    x[M // 2] = 0.0
    tc, plain = torch.empty(M, N, device=DEV), torch.empty(M, N, device=DEV)
    assert run(x, w, tc, M)
    B.gemm_plain(x, w, plain, M, 0, B.stream_ptr())
    ref = x.double() @ w.double().t()
    # every single output: K rounded additions, each at most 2^-24 of the sum of magnitudes (and 2^-149 where that is subnormal)
    bound = 1024 * (2.0 ** -24 * (x.double().abs() @ w.double().abs().t()) + 2.0 ** -149)
    assert ((tc - ref).abs() <= bound).all()
    assert (tc - ref).norm() <= 1.1 * (plain - ref).norm()
    assert (tc[M // 2] == 0).all()
    if exponent <= -80:
        assert ((tc == plain) | (tc == 0)).all() and (tc == 0).sum() <= N + 10       # (a sum may cancel to 0, which stays)
        both = torch.randn(M, N, device=DEV) * 2.0 ** exponent
        total = both.clone()
        assert run(x, w, total, M, mode=1)
        assert torch.equal(total, both + tc)
