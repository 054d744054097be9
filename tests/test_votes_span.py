"""The vote kernel's launches, without a GPU: its tiles of 256 samples x 240 clause
rows are counted in 32 bits, and a CTA pair's tile number steps once past the end,
so a launch stays below 2^31 tiles."""
import ctypes

import pytest


@pytest.mark.parametrize("rows", [8, 240, 241, 5120, 40960, 262144, 7864320, (1 << 31) - 8])
def test_tiles_of_a_launch_fit_their_counter(rows):
    import santoku_tsetlin as tm
    span_of = tm.lib().tmb_votes_span
    span_of.restype, span_of.argtypes = ctypes.c_uint32, [ctypes.c_uint64]
    span = span_of(rows)
    row_tiles = -(-rows // 240)
    for n in (1, 256, 257, (1 << 25) + 3, (1 << 31) - 1):
        first = min(n, span)
        assert first == n or first % 256 == 0
        assert -(-first // 256) * row_tiles < 1 << 31
    # the sizes in use take one launch: 2^31 tiles are 1.3e14 sample and clause pairs
    assert span >= min((1 << 31) - 1, (1 << 45) // (row_tiles * 240))
