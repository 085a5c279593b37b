"""Products of few tokens whose K is shared by the CTAs of a cluster, at the sizes where the sharing can go wrong: one tile
of rows and several, a last tile that is not full, parts of unequal length, every width of the token tile.

Tolerance: one rounding to bfloat16 (2^-9 of a value, 6e-3 of the largest with the activation's own, as elsewhere)."""

import pytest
import torch

DEV = "cuda:0"
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [1, 16, 17, 64])
@pytest.mark.parametrize("N, K", [(32, 512), (128, 520), (160, 1096), (1024, 2048), (2080, 4160), (4736, 1024)])
def test_products_by_parts(N, K, T):
    from llmoxide_b200 import kernels
    torch.manual_seed(N + K + T)
    x, w = torch.randn(T, K, device=DEV).bfloat16(), (torch.randn(N, K, device=DEV) * K ** -0.5).bfloat16()
    want = x.double() @ w.double().T
    rel = lambda a, b: ((a.double() - b).abs().max() / b.abs().max()).item()
    out = torch.full((T, N), 7.0, device=DEV).bfloat16()
    kernels.gemm_tc(x, w, out)
    assert rel(out, want) < 6e-3
    kernels.gemm_tc(x, w, out, gated=3, activation="relu_squared")
    assert rel(out, torch.relu(want) ** 2) < 1.2e-2
    if N % 32 == 0:
        blocks = want.view(T, N // 32, 2, 16)
        act = torch.nn.functional.silu(blocks[:, :, 0]) * blocks[:, :, 1]
        half = torch.empty(T, N // 2, device=DEV, dtype=torch.bfloat16)
        kernels.gemm_tc(x, w, half, gated=2)
        assert rel(half, act.reshape(T, N // 2)) < 6e-3
        # with a norm's row scales: the second half of an RMS norm over x
        sumsq = torch.randn(3, 64, device=DEV).abs()
        r = 1.0 / torch.sqrt(sumsq[:, :T].double().sum(0) / K + 1e-6)
        act = torch.nn.functional.silu(blocks[:, :, 0] * r[:, None, None]) * blocks[:, :, 1] * r[:, None, None]
        kernels.gemm_tc(x, w, half, gated=2, scale=(sumsq, 3, 1e-6, K))
        assert rel(half, act.reshape(T, N // 2)) < 6e-3
    assert kernels.gemm_tc_status() == 0
