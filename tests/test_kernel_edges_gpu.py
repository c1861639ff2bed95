"""Sizes at which the work split of the kernels changes: tile edges, remainders, smallest and largest of a range, against the
oracle (bit for bit: moved rows, and sums whose order and roundings the contract fixes)."""
import pytest

from test_ll_gpu import _case as ll_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("world,tokens,hidden,experts,topk,mode", [
    (1, [1], 7168, 256, 8, 2),              # one token: its row is cut into as many pieces as it has groups of 128 values
    (1, [256], 136, 8, 3, 0),               # the last group of a row is short
    (1, [33], 128, 1, 1, 1),                # a single group, a single expert
    (1, [250], 8192, 1000, 9, 2),           # several pieces of a row per warp, more experts than layout threads
    (2, [1, 256], 384, 1024, 8, 2),         # the most experts; own rows next to rows of a peer
    (4, [255, 0, 1, 32], 640, 8, 6, 0),
    (8, [9, 64, 65, 1, 31, 33, 2, 128], 1152, 64, 8, 1),
])
def test_low_latency_splits(world, tokens, hidden, experts, topk, mode):
    ll_case(world, tokens, hidden, experts, topk, mode, routes="invalid", repeats=3)
