"""The gated expert products on both sides of the rule that picks their row tiles."""

import pytest
import torch

DEV = "cuda:0"
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E, top, F, T", [(16, 2, 1024, 4), (16, 2, 1000, 1), (64, 4, 512, 16), (64, 4, 512, 100),
                                          (8, 2, 3000, 16), (4, 1, 72, 64), (32, 2, 136, 250)])
def test_gated_expert_products(E, top, F, T):
    """One rounding to bfloat16 (2^-9 of a value, 6e-3 of the largest with the activation's own, as elsewhere)."""
    from llmoxide_b200 import kernels
    torch.manual_seed(E + F + T)
    K, P = 264, T * top
    w = (torch.randn(E, 2 * F, K, device=DEV) * K ** -0.5).bfloat16()
    ids = torch.stack([torch.randperm(E)[:top] for _ in range(T)]).int().to(DEV)
    perm, dest = (torch.empty(P, dtype=torch.int32, device=DEV) for _ in range(2))
    tiles = torch.empty(kernels.moe_max_tiles(P, E, 16), 3, dtype=torch.int32, device=DEV)
    sw, pw = torch.empty(P, device=DEV), torch.rand(T, top, device=DEV)
    kernels.moe_sort(ids, E, perm, tiles, 16, pw, dest, sw)
    x = torch.randn(T, K, device=DEV).bfloat16()
    xs, y = torch.empty(P, K, dtype=torch.bfloat16, device=DEV), torch.full((P + 1, F), 7.0, device=DEV).bfloat16()
    kernels.moe_gather_rows(x, perm, top, xs)
    kernels.moe_grouped_tc(xs, w, y[:P], tiles, 16, dest, sw, gated=1)
    torch.cuda.synchronize()
    kernels.check_status()
    expert = ids.flatten()[perm.long()]
    gu = torch.stack([xs[i].double() @ w[expert[i]].double().T for i in range(P)])
    want = torch.nn.functional.silu(gu[:, :F]) * gu[:, F:]
    assert ((y[:P].double() - want).abs().max() / want.abs().max()).item() < 6e-3 and (y[P] == 7.0).all()
