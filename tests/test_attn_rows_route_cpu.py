"""Which heads the tcgen05 attention over runs of rows takes: rows of keys and values that are whole boxes of 64 columns; other heads of up to
128 entries take the mma.sync kernel with the same weights."""
import ctypes

import pytest

from conftest import pkg


@pytest.mark.parametrize("heads,kv,dim,vdim,bs,takes", [
    (16, 4, 128, 128, 128, 1), (8, 2, 64, 64, 64, 1), (8, 2, 64, 128, 128, 1), (8, 2, 128, 64, 192, 1), (16, 1, 64, 64, 64, 1), (1, 1, 128, 128, 64, 1),
    (6, 2, 64, 32, 128, 2), (6, 2, 32, 64, 128, 2), (3, 3, 32, 48, 64, 2), (16, 1, 80, 48, 128, 2), (10, 2, 96, 128, 192, 2), (8, 2, 128, 112, 128, 2),
    (32, 32, 16, 16, 64, 2), (8, 2, 192, 128, 128, 0), (8, 2, 128, 256, 128, 0), (17, 1, 64, 64, 64, 0), (6, 4, 64, 64, 64, 0), (8, 2, 64, 64, 96, 0), (8, 2, 72, 64, 64, 0)])
def test_heads_of_whole_boxes(heads, kv, dim, vdim, bs, takes):
    f = pkg("_abi").lib().b200_debug_attn_rows_tc
    f.argtypes = [ctypes.c_int32] * 5
    assert f(heads, kv, dim, vdim, bs) == takes
