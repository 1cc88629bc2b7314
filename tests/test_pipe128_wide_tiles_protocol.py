"""The barriers of the D = 128 backward without tangents: one ring of both loop tensors whichever side is the CTA's own, released by both issuing
threads; a group of elementwise threads for each 16 columns of a tile of 64 queries or 96 keys."""
import pytest

from tests.test_pipe128_barrier_protocol import run_backward


@pytest.mark.parametrize("groups", [4, 6], ids=["own_keys", "own_queries"])
def test_no_deadlock_and_no_premature_pass(groups):
    """(With own queries there are no statistics to wait for; the model's arrive at once.)"""
    for n_tiles in (1, 2, 3, 4, 5, 9, 32):
        for seed in range(10):
            assert run_backward(n_tiles, True, groups, seed) == "ok", (n_tiles, seed)
