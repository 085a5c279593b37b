"""The router's product around the numbers of rows at which a warp takes one, two or more of them."""

import pytest
import torch

DEV = "cuda:0"
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [1, 3, 500])
@pytest.mark.parametrize("n_rows", [6, 8, 9, 16, 17, 24, 25, 33])
@pytest.mark.parametrize("K, dtype", [(512, torch.bfloat16), (264, torch.float32), (100, torch.float32)])
def test_router_products(T, n_rows, K, dtype):
    """Rows behind the experts' go out as they are.  float32 sums of up to 512 products in 32 chains: 1e-6 of the root of
    their number; a row's bits do not depend on where it lies."""
    from llmoxide_b200 import kernels
    torch.manual_seed(n_rows * T)
    x, w = torch.randn(T, K, device=DEV).to(dtype), torch.randn(n_rows, K, device=DEV)
    E = 4
    w[:E] *= K ** -0.5                     # (scores that are told apart)
    ids, weights = torch.empty(T, 2, dtype=torch.int32, device=DEV), torch.empty(T, 2, device=DEV)

    def run(w):
        out = torch.empty(T, n_rows - E, device=DEV)
        kernels.moe_router(x, w, ids, weights, 1, 1, 1, "sigmoid", False, 0.0, 1.0, extra_out=out)
        return out

    out, want = run(w), x.double() @ w.double().T
    assert ((out - want[:, E:]).abs().max() / K ** 0.5).item() < 1e-6
    top = torch.sigmoid(want[:, :E]).topk(2, 1)
    assert torch.equal(ids.long(), top.indices) and ((weights - top.values).abs() < 1e-5).all()
    order = torch.randperm(n_rows - E, device=DEV)
    assert torch.equal(run(torch.cat([w[:E], w[E:][order]])), out[:, order])
