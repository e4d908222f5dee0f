"""The rule for the tiles that change between channels-first and channels-last memory (``csrc/pad.cu``), asked on the host
for a GPU of 148 SMs, which is what the library assumes without one."""
import ctypes

import pytest

from distdl_b200 import _native

pytestmark = pytest.mark.skipif(not _native.available(), reason="native library not built")


@pytest.mark.parametrize("to_last,B,C,size,words", [
    (1, 1, 8, 82, 32), (1, 8, 8, 82, 32), (1, 4, 24, 122, 32), (1, 1, 16, 242, 32),      # few CTAs: the widest tile into
    (1, 8, 8, 122, 4), (1, 4, 24, 162, 8), (1, 8, 16, 162, 8), (1, 8, 40, 162, 8), (1, 8, 64, 162, 32), (1, 8, 96, 162, 16),
    (0, 1, 8, 82, 4), (0, 1, 24, 82, 8), (0, 1, 64, 82, 32)])                              # ... but not back
def test_narrow_tiles_where_there_are_ctas_enough(to_last, B, C, size, words):
    assert _native.lib().dd_shift_channels_words(to_last, B, C, ctypes.c_longlong(size * size)) == words
