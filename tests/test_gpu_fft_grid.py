"""
Grids of the mixed-radix FFT passes: the blocks that fit on an SM depend on the line's shared memory, so a length gets the
same grid whichever lengths the process transformed before.
"""
import pytest

pytestmark = pytest.mark.gpu


def test_blocks_follow_the_line_length():
    from pyrecon_b200 import _lib as L
    blocks = L.load().prc_debug_fft_strided_blocks
    # 80 registers let three blocks of 256 threads on an SM; tiles of 26, 72 and 60 KB leave room for three, one of 2000
    # points (two lines, 80 KB) for two
    lengths, expected = [100, 1000, 2000, 1500], [3, 3, 2, 3]
    assert [blocks(n, 4) for n in lengths] == expected
    assert [blocks(n, 4) for n in reversed(lengths)] == expected[::-1]
