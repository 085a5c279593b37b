"""What a parallel block hands to whoever follows it, on the CPU."""

from types import SimpleNamespace

import pytest
import torch

from llmoxide_b200.parts.block import ParallelBlock
from llmoxide_b200.parts.norm import Joined, LayerNorm, RMSNorm, WeightedSum


class Part:
    """A norm, mixer or feed-forward that hands out what it was made with and notes what it was given."""

    def __init__(self, result, adds=False):
        self.result, self.added, self.residuals, self.adds_to_residual = result, [], [], adds

    def add(self, h, delta):
        self.added.append(delta)

    def add_forward(self, h, delta):
        return h

    def add_forward_pair(self, h, delta, other):
        return h, h

    def forward(self, *args, residual=None):
        self.residuals.append(residual)
        return self.result


def block_of(a, out, norms="one", adds=False):
    block = ParallelBlock.__new__(ParallelBlock)
    block.rt = SimpleNamespace(shared={}, device="cpu")
    block.norm, block.mixer_norm, block.ff_norm = (Part(None), None, None) if norms == "one" else (None, Part(None), Part(None))
    block.mixer, block.feed_forward = Part(a, adds), Part(out, adds)
    return block


def test_results_are_joined_where_both_are_tensors_and_the_follower_takes_them():
    h, ctx = torch.zeros(2, 8), SimpleNamespace(probe=None)
    a, out = torch.ones(2, 8), torch.ones(3, 2, 8)
    weighted = WeightedSum([(a, 0.5), (a, 2.0)])
    for joins, mixed in ((True, a), (False, a), (True, weighted), (False, weighted), (True, None)):
        block = block_of(mixed, out)
        block.joins_results = joins
        pending = block.forward(h, None, ctx, None)
        if joins and mixed is a:
            assert isinstance(pending, Joined) and pending.terms == [a, out] and not block.norm.added
        else:
            assert pending is out and block.norm.added == ([] if mixed is None else [mixed])


def test_a_branch_leaves_the_stream_to_the_mixer(monkeypatch):
    """Parts that add to the stream where they are given it: one after the other both are, side by side one is."""
    from llmoxide_b200 import kernels
    from llmoxide_b200.parts import branches
    assert branches.MAX_TOKENS <= kernels.PAIR_MIN_TOKENS         # (products of more tokens add to the stream themselves)
    h, a, out = torch.zeros(2, 8), torch.ones(2, 8), torch.ones(2, 8)
    monkeypatch.setattr(branches, "fork", lambda rt, name, work: (work(), lambda: None))
    for side_by_side in (False, True):
        monkeypatch.setattr(branches, "wanted", lambda ctx, n: side_by_side)
        block = block_of(a, out, norms="two", adds=True)
        pending = block.forward(h, None, SimpleNamespace(probe=None), None)
        assert pending.terms == [a, out] and block.mixer.residuals == [h]
        assert block.feed_forward.residuals == ([None] if side_by_side else [h])


def rms_norm(size):
    norm = RMSNorm.__new__(RMSNorm)
    norm.size = size
    return norm


@pytest.mark.parametrize("final, streams, joins", [
    (rms_norm(2048), 1, True), (rms_norm(50), 1, False), (rms_norm(8196), 1, False), (LayerNorm.__new__(LayerNorm), 1, False),
    (Part(None), 1, False), (rms_norm(2048), 2, False)])
def test_followers_that_take_joined_results(final, streams, joins):
    """Every call behind one of a block's counts: here the block itself, another one and the model's last norm."""
    from llmoxide_b200.parts.block import join_results
    blocks = [block_of(None, None), block_of(None, None)]
    for block in blocks:
        block.norm = rms_norm(64)
    calls = [SimpleNamespace(layer=i) for i in (0, 0, 1)]
    join_results(blocks, calls, final, streams)
    assert [b.joins_results for b in blocks] == [streams == 1, joins]
    join_results(blocks, calls + calls[:1], final, streams)
    assert [b.joins_results for b in blocks] == [joins, streams == 1]
    blocks[1] = object()                                   # a block of another arrangement says nothing
    join_results(blocks, calls, final, streams)
    assert not blocks[0].joins_results
