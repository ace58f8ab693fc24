"""Several products of equal sizes in one launch, and products of few outputs in the token tiles they are given, against fp32 sums of the
same bfloat16 operands."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("M,N,K,batches", [(257, 256, 64, 4), (300, 512, 200, 2), (1000, 256, 520, 3), (384, 768, 128, 1)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_batched_product(M, N, K, batches, dtype):
    from inference_engine_rust_b200.csrc import bindings as B
    g = torch.Generator(device=DEV).manual_seed(M + N)
    rows = M + 7                                                    # rows of other tokens between the products' inputs
    x = torch.randn((batches + 1, rows, K), generator=g, device=DEV).bfloat16()
    w = torch.randn((batches * N, K), generator=g, device=DEV).bfloat16()
    out = torch.full((M + 2, batches * N + 8), 7.0, dtype=dtype, device=DEV)
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    assert B.gemm_tc_batched(x[:batches], w, out, M, batches, err, B.stream_ptr())
    assert err.item() == 0
    want = torch.cat([x[b, :M].double() @ w[b * N:(b + 1) * N].double().t() for b in range(batches)], dim=1)
    # fp32 sums of K products, each at most 2^-24 of the sum of magnitudes off per step; bfloat16 results round once more
    size = torch.cat([x[b, :M].double().abs() @ w[b * N:(b + 1) * N].double().abs().t() for b in range(batches)], dim=1)
    got = out[:M, :batches * N].double()
    assert ((got - want).abs() <= size * K * 2.0 ** -24 + (want.abs() * 2.0 ** -8 if dtype == torch.bfloat16 else 0)).all()
    assert (out[M:] == 7).all() and (out[:M, batches * N:] == 7).all()


def test_batched_product_refuses():
    from inference_engine_rust_b200.csrc import bindings as B
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    w = torch.zeros((512, 64), dtype=torch.bfloat16, device=DEV)
    out = torch.zeros((300, 512), device=DEV)
    x = torch.zeros((2, 300, 64), dtype=torch.bfloat16, device=DEV)
    assert not B.gemm_tc_batched(x, w, out, 256, 2, err, B.stream_ptr())            # few tokens
    assert not B.gemm_tc_batched(x, w[:500], out, 300, 2, err, B.stream_ptr())      # outputs that share a tile


@pytest.mark.parametrize("N,K", [(64, 1024), (288, 512), (130, 72)])
@pytest.mark.parametrize("M", [129, 256, 257, 1000, 2100])
def test_few_outputs(M, N, K):
    from inference_engine_rust_b200.csrc import bindings as B
    from inference_engine_rust_b200.parts import Runtime
    from inference_engine_rust_b200.parts.linear import Linear
    g = torch.Generator(device=DEV).manual_seed(M + N)
    rt = Runtime(dtype=torch.bfloat16, device=torch.device(DEV))
    x = torch.randn((M, K), generator=g, device=DEV).bfloat16()
    w = torch.randn((N, K), generator=g, device=DEV).bfloat16()
    out = torch.full((M + 1, N), 7.0, device=DEV)
    Linear(w, rt, narrow=True).apply(x, out, M, B.stream_ptr())
    assert rt.err.item() == 0
    size = x.double().abs() @ w.double().abs().t()
    assert ((out[:M].double() - x.double() @ w.double().t()).abs() <= size * K * 2.0 ** -24).all()      # as above
    assert (out[M:] == 7).all()
