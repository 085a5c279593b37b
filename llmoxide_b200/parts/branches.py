"""Branches of a captured decode step.

A decode step is a chain of short kernels, each of which waits for the one before; where two parts of a layer read the same
rows and not one another's results, their chains can be branches of the step's graph.  A branch is captured on a stream of
its own that the model keeps: forked behind what was launched so far, joined by the caller ahead of whatever reads its
results.  What a branch allocates is used again by its own stream only, and whoever forks holds what crosses over (the rows
that are read, the results) until the join.  Steps that are launched one by one are not cut up: their allocations would need
the streams' events, and their launches are what they wait for.
"""

from __future__ import annotations

import torch

# The most tokens of a step that is cut up.  Two designs' steps (parallel blocks, most with routed experts; prompts of 200
# tokens behind them) as one chain and in branches, us: 1 token 415 and 343, 516 and 378; 8: 544 and 511, 588 and 503; 16: 610
# and 571, 677 and 583; 32: 689 and 652, 828 and 704; 64: 874 and 831, 1036 and 887.  Longer steps were not tried.
MAX_TOKENS = 64


def wanted(ctx, n_tokens: int) -> bool:
    return bool(getattr(ctx, "is_decode", False) and n_tokens <= MAX_TOKENS and torch.cuda.is_current_stream_capturing())


def fork(rt, name: str, work):
    """(``work()``, captured on the model's stream ``name``; the function that joins it)."""
    here = torch.cuda.current_stream()
    side = rt.shared.get(("stream", name))
    if side is None:
        side = rt.shared[("stream", name)] = torch.cuda.Stream(device=rt.device)
    side.wait_stream(here)
    with torch.cuda.stream(side):
        out = work()
    return out, lambda: here.wait_stream(side)
