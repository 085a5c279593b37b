"""Long prompts of the linear attention by chunks, at the sizes where they can go wrong: around a chunk's and a tile's
edge, sizes that are no multiple of four, short sequences beside long ones.

Tolerance: an output is a sum of at most three chains of 128 multiply-adds and the state a sum per chunk, with normal
entries whose rounding errors are independent: 5e-7 of the 64-bit result in the 2-norm (2^-24 times the root of 64)."""

import pytest
import torch

DEV = "cuda:0"
pytestmark = pytest.mark.gpu


def run(proj, lens, H, D, Dv, decay, state, slots):
    from llmoxide_b200 import kernels
    starts = torch.tensor([sum(lens[:i]) for i in range(len(lens) + 1)], dtype=torch.int32, device=DEV)
    pos = torch.cat([torch.arange(n, dtype=torch.int32) for n in lens]).to(DEV)
    out = torch.full((sum(lens), H * Dv), float("nan"), device=DEV)
    kernels.decay_scan(proj, out, state, starts, pos, torch.tensor(slots, dtype=torch.int32, device=DEV), decay, None, None, 0,
                       "none", 1.0, H, D, Dv, 0, H * D, 2 * H * D, max_new=max(lens))
    return out


@pytest.mark.parametrize("H, D, Dv", [(2, 64, 64), (3, 68, 70), (1, 128, 65), (2, 128, 128), (1, 200, 66), (1, 256, 256)])
def test_chunks_against_64_bits(H, D, Dv):
    torch.manual_seed(D + Dv)
    lens, slots = [129, 1, 192, 64, 193, 257, 128], [5, 0, 3, 1, 7, 2, 6]
    decay = torch.tensor([0.9, 1.0, 0.999][:H], device=DEV)
    proj = torch.randn(sum(lens), H * (2 * D + Dv), device=DEV)
    before = torch.randn(8, H, D, Dv, device=DEV)
    state = before.clone()
    out = run(proj, lens, H, D, Dv, decay, state, slots)
    assert torch.equal(state[4], before[4])                       # no sequence's
    t0, g = 0, decay.double()[:, None, None]
    for n, slot in zip(lens, slots):
        p = proj[t0 : t0 + n].double()
        q, k, v = p[:, : H * D].view(n, H, D), p[:, H * D : 2 * H * D].view(n, H, D), p[:, 2 * H * D :].view(n, H, Dv)
        S, want = before[slot].double(), []
        for t in range(n):
            S = g * S + k[t, :, :, None] * v[t, :, None, :]
            want.append((q[t, :, :, None] * S).sum(1).reshape(-1))
        want = torch.stack(want)
        assert ((out[t0 : t0 + n] - want).norm() / want.norm()).item() < 5e-7, n
        assert ((state[slot] - S).norm() / S.norm()).item() < 5e-7, n
        # a sequence's result does not depend on its neighbours, whichever way it goes
        alone = before.clone()
        assert torch.equal(run(proj[t0 : t0 + n], [n], H, D, Dv, decay, alone, [slot]), out[t0 : t0 + n])
        assert torch.equal(alone[slot], state[slot])
        t0 += n


@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("at", [64, 70, 100, 127, 130])
def test_a_value_that_is_not_finite_changes_no_token_before_it(at, bad):
    H, D, Dv, n = 2, 128, 65, 140
    torch.manual_seed(at)
    decay, proj = torch.tensor([0.9, 0.99], device=DEV), torch.randn(n, H * (2 * D + Dv), device=DEV)
    start = torch.randn(1, H, D, Dv, device=DEV)
    clean = run(proj, [n], H, D, Dv, decay, start.clone(), [0])
    proj[at, 2 * H * D + 3] = bad                                  # head 0, column 3
    state = start.clone()
    out = run(proj, [n], H, D, Dv, decay, state, [0])
    changed = torch.zeros(n, H * Dv, dtype=torch.bool, device=DEV)
    changed[at:, 3] = True
    assert torch.equal(~torch.isfinite(out), changed)
    assert torch.equal(out[~changed], clean[~changed])
    lost = torch.zeros(H, D, Dv, dtype=torch.bool, device=DEV)
    lost[0, :, 3] = True
    assert torch.equal(~torch.isfinite(state[0]), lost)
