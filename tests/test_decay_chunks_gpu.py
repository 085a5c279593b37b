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


@pytest.mark.parametrize("at", [64, 70, 100, 127, 130])
def test_a_value_at_the_end_of_the_range_reaches_its_own_column_only(at):
    """The largest finite values are values like others: finite results, and the tokens before one keep their bits."""
    H, D, Dv, n = 2, 128, 65, 140
    torch.manual_seed(at)
    decay, proj = torch.tensor([0.9, 0.99], device=DEV), torch.randn(n, H * (2 * D + Dv), device=DEV)
    proj[at, H * D : 2 * H * D] *= 0.01                            # (keys below 1: sums of the products stay in range)
    start = torch.randn(1, H, D, Dv, device=DEV)
    clean = run(proj, [n], H, D, Dv, decay, start.clone(), [0])
    proj[at, 2 * H * D + 3] = 3.4025e38                            # head 0, column 3
    state = start.clone()
    out = run(proj, [n], H, D, Dv, decay, state, [0])
    changed = torch.zeros(n, H * Dv, dtype=torch.bool, device=DEV)
    changed[at:, 3] = True
    assert torch.equal(out[~changed], clean[~changed])
    assert torch.isfinite(out).all() and torch.isfinite(state).all()


def test_products_of_equal_operands():
    """Operands that are all (1 + 2^-11 - 2^-23) or its negative, whose products lose the same way every time where an
    operand is cut in parts that do not hold all its bits.  Tolerance as above."""
    H, D, Dv, n, e = 1, 128, 128, 192, 1 + 2.0 ** -11 - 2.0 ** -23
    torch.manual_seed(0)
    proj = torch.where(torch.rand(n, H * (2 * D + Dv), device=DEV) < 0.5, -e, e)
    decay, before = torch.tensor([1.0], device=DEV), torch.zeros(1, H, D, Dv, device=DEV)
    state = before.clone()
    out = run(proj, [n], H, D, Dv, decay, state, [0])
    one = torch.ones(n, H, device=DEV, dtype=torch.float64)
    want, after = recurrence(proj, [n], [0], before, one, one, H, D, Dv, False)
    assert ((out - want).norm() / want.norm()).item() < 5e-7
    assert ((state - after).norm() / after.norm()).item() < 5e-7


def recurrence(proj, lens, slots, state, a, b, H, D, Dv, ones):
    """Token by token in 64 bits; a, b: [T, H]."""
    outs, t0 = [], 0
    after = state.double()
    for n, slot in zip(lens, slots):
        p = proj[t0 : t0 + n].double()
        q, k, v = p[:, : H * D].view(n, H, D), p[:, H * D : 2 * H * D].view(n, H, D), p[:, 2 * H * D : 2 * H * D + H * Dv].view(n, H, Dv)
        if ones:
            v = torch.cat([v, torch.ones(n, H, 1, device=DEV, dtype=torch.float64)], 2)
        S = after[slot].clone()
        for t in range(n):
            S = a[t0 + t, :, None, None] * S + b[t0 + t, :, None, None] * k[t, :, :, None] * v[t, :, None, :]
            outs.append((q[t, :, :, None] * S).sum(1).reshape(-1))
        after[slot] = S
        t0 += n
    return torch.stack(outs), after


@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("H, D, Dv, lens", [
    (2, 32, 30, [300, 40]), (1, 30, 31, [129, 127, 1]),            # small states: one pass or two of two columns
    (2, 128, 65, [100] * 6), (1, 66, 40, [128] * 4 + [64]),         # many prompts of up to a segment
    (1, 64, 33, [257, 300]), (2, 128, 64, [270]),                   # longer than two segments
    (1, 130, 20, [300]), (1, 256, 16, [140, 3]), (1, 192, 20, [650])])    # keys above 128: one column, two in long prompts
def test_one_and_two_columns_a_thread(H, D, Dv, lens, gated):
    """Prompts by two columns a thread against 64 bits, and the same prompts one token a step, which one column takes:
    up to a segment the same bits.  Tolerance as above (up to 256 multiply-adds a chain: 1e-6)."""
    from llmoxide_b200 import kernels
    torch.manual_seed(D + Dv)
    T, B, slots, dva = sum(lens), len(lens), list(range(len(lens)))[::-1], Dv + int(gated)
    proj = torch.randn(T, H * (2 * D + Dv), device=DEV)
    decay = torch.tensor([0.9, 0.999][:H], device=DEV)
    before = torch.randn(B, H, D, dva, device=DEV)
    ab = torch.rand(2, T, H, device=DEV) * 0.3 + 0.69 if gated else None
    seg_of = torch.cat([torch.arange(n) // 128 for n in lens])

    def call(rows, n_of, state, seqs):
        """``rows`` of every sequence in ``seqs``, n_of tokens each."""
        starts = torch.tensor([sum(n_of[:i]) for i in range(len(seqs) + 1)], dtype=torch.int32, device=DEV)
        out = torch.full((len(rows), H * dva), float("nan"), device=DEV)
        gates = None
        if gated:
            gates = torch.empty(len(rows), H, 4, device=DEV)
            gates[:, :, 0], gates[:, :, 1], gates[:, :, 2] = ab[0, rows], ab[1, rows], 1.0
            t0 = 0
            for n in n_of:                                          # the product of a over the token's segment so far
                for s in range(0, n, 128):
                    gates[t0 + s : t0 + min(n, s + 128), :, 3] = ab[0, rows][t0 + s : t0 + min(n, s + 128)].cumprod(0)
                t0 += n
        kernels.decay_scan(proj[rows], out, state, starts, torch.zeros(len(rows), dtype=torch.int32, device=DEV),
                           torch.tensor([slots[b] for b in seqs], dtype=torch.int32, device=DEV), None if gated else decay,
                           None, None, 0, "none", 1.0, H, D, Dv, 0, H * D, 2 * H * D, max_new=max(n_of), gates=gates,
                           ones_column=gated)
        return out

    state = before.clone()
    out = call(torch.arange(T, device=DEV), lens, state, list(range(B)))
    a = ab[0].double() if gated else decay.double().expand(T, H)
    b = ab[1].double() if gated else torch.ones(T, H, device=DEV, dtype=torch.float64)
    want, after = recurrence(proj, lens, slots, before, a, b, H, D, Dv, gated)
    assert ((out - want).norm() / want.norm()).item() < 1e-6
    assert ((state - after).norm() / after.norm()).item() < 1e-6
    if max(lens) <= 128:
        alone = before.clone()
        starts = [sum(lens[:b]) for b in range(B)]
        for t in range(max(lens)):
            seqs = [b for b in range(B) if t < lens[b]]
            rows = torch.tensor([starts[b] + t for b in seqs], device=DEV)
            assert torch.equal(call(rows, [1] * len(seqs), alone, seqs), out[rows])
        assert torch.equal(alone, state)


@pytest.mark.parametrize("H, D, Dv, n_rot, activation, ones", [
    (2, 66, 65, 0, "none", False), (1, 131, 64, 0, "none", False),          # keys that are no multiple of four
    (2, 128, 64, 128, "silu", False), (1, 70, 66, 32, "none", False),       # rotated, all of a key or its first dims
    (2, 64, 64, 0, "none", True), (1, 67, 63, 10, "silu", True)])           # one more column, of ones
def test_chunks_of_prepared_keys_and_values(H, D, Dv, n_rot, activation, ones):
    """As above; an activation and a rotation add a few roundings of 2^-24 to every q, k and v: 7e-7 in the 2-norm."""
    from llmoxide_b200 import kernels
    torch.manual_seed(D + Dv)
    lens, slots, dva = [150, 1, 193], [1, 3, 0], Dv + int(ones)
    decay = torch.tensor([0.95, 0.999][:H], device=DEV)
    T, before = sum(lens), torch.randn(4, H, D, dva, device=DEV)
    proj = torch.randn(T, H * (2 * D + Dv), device=DEV)
    starts = torch.tensor([sum(lens[:i]) for i in range(4)], dtype=torch.int32, device=DEV)
    pos = torch.cat([torch.arange(7, 7 + n, dtype=torch.int32) for n in lens]).to(DEV)
    angle = torch.rand(max(lens) + 7, n_rot // 2, device=DEV) * 6.28 if n_rot else None
    cos, sin = (angle.cos(), angle.sin()) if n_rot else (None, None)
    state, out = before.clone(), torch.full((T, H * dva), float("nan"), device=DEV)
    kernels.decay_scan(proj, out, state, starts, pos, torch.tensor(slots, dtype=torch.int32, device=DEV), decay, cos, sin,
                       n_rot, activation, 0.7, H, D, Dv, 0, H * D, 2 * H * D, max_new=max(lens), q_scale=1.3, ones_column=ones)
    p = torch.nn.functional.silu(proj.double()) if activation == "silu" else proj.double()
    q, k, v = p[:, : H * D].view(T, H, D), p[:, H * D : 2 * H * D].view(T, H, D), p[:, 2 * H * D :]
    if n_rot:
        half, c, s = n_rot // 2, cos.double()[pos.long()][:, None], sin.double()[pos.long()][:, None]
        q, k = (torch.cat([z[..., :half] * c - z[..., half:n_rot] * s, z[..., half:n_rot] * c + z[..., :half] * s, z[..., n_rot:]], 2)
                for z in (q, k))
    prepared = torch.cat([q.reshape(T, -1) * 1.3, k.reshape(T, -1) * 0.7, v], 1)
    one = torch.ones(T, H, device=DEV, dtype=torch.float64)
    want, after = recurrence(prepared, lens, slots, before, one * decay.double(), one, H, D, Dv, ones)
    assert ((out - want).norm() / want.norm()).item() < 7e-7
    assert ((state - after).norm() / after.norm()).item() < 7e-7
