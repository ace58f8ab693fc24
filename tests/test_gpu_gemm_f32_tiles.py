"""The fp32 projection on the tensor cores in tiles of 80, 96, 112 and 128 tokens: against 64-bit products, and a row's bits whatever the tile."""
import pytest
import torch

from test_gpu_gemm_f32 import DEV, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [66, 80, 81, 96, 97, 112, 113, 128, 161, 222, 333, 400])
@pytest.mark.parametrize("N,K", [(136, 1024), (4100, 1060), (200, 4096)])
def test_tiles(M, N, K):
    g = torch.Generator(device=DEV).manual_seed(M + N)
    x, w = torch.randn((M, K), generator=g, device=DEV), torch.randn((N, K), generator=g, device=DEV)
    out = torch.full((M + 1, N), 5.0, device=DEV)
    assert run(x, w, out, M)
    ref = x.double() @ w.double().t()
    # K / 64 rounded additions and twelve truncating ones per 64 k, each at most 2^-23 of the sum of magnitudes it meets
    assert ((out[:M] - ref).abs() <= 2.0 ** -19 * (x.double().abs() @ w.double().abs().t())).all()
    assert (out[M] == 5.0).all()
    few = torch.empty((40, N), device=DEV)
    assert run(x[M - 40:], w, few, 40)
    assert torch.equal(few, out[M - 40:M])
