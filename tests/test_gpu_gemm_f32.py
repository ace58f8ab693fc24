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
