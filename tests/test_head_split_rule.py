"""Over how many parts of K the head's input gradient is split."""
import pytest

from levanter_b200.ops.cross_entropy import GRAD_BYTES, _dx_splits


@pytest.mark.parametrize("tiles,k_blocks,rows,cols,want", [
    (48, 1572, 4096, 768, {3}),        # 48 tiles leave a third of the pairs idle: 144 pieces are two whole waves
    (248, 1572, 7936, 2048, {1, 2, 3}),  # nearly whole waves as it is: a fraction of a wave is not worth 65 MB of sums per split, five times
    (74, 1572, 4736, 1024, {1}),       # one whole wave
    (2, 40, 257, 256, {2}),            # at least 16 blocks each
    (1, 3, 64, 64, {1}),
])
def test_splits(tiles, k_blocks, rows, cols, want):
    assert _dx_splits(tiles, k_blocks, 74, 4 * rows * cols) in want


def test_sums_are_bounded():
    for out_bytes in (GRAD_BYTES // 3, GRAD_BYTES, 4 * GRAD_BYTES):
        s = _dx_splits(10, 100000, 74, out_bytes)
        assert s == 1 or s * out_bytes <= GRAD_BYTES
