"""Which fp8 products take the 128x256 tiles: those that save the persistent grid a turn."""
import pytest

from hyper_parallel_b200.ops.fp8 import _wide_tiles


@pytest.mark.parametrize("M,N,wide", [
    (128, 256, False), (700, 1536, False), (128 * 148, 128, False),       # one turn with the small tiles
    (20000, 64, False), (20000, 128, False), (40000, 8, False),           # at most half of a wide tile in use
    (4096, 1152, False),                                                  # two turns either way
    (4096, 640, True), (128 * 149, 256, True), (20000, 384, True), (4096, 36864, True), (16, 40000, True),
    (4096, 644, False)])                                                  # rows that are not whole vectors
def test_rule(M, N, wide):
    assert _wide_tiles(M, N, 148) is wide
