"""Which kernels take a step of matrix memory: segments only where all of their clusters (of four CTAs, one an SM) run at a time and,
where the rows of the step are known, one portion may be long enough for them."""
import ctypes

import pytest

from conftest import pkg

WALK, CHUNKS, SEGMENTS = 0, 1, 2


@pytest.mark.parametrize("seqs,heads,dim,vdim,want", [
    (1, 8, 128, 256, SEGMENTS), (2, 4, 128, 256, SEGMENTS), (4, 2, 64, 256, SEGMENTS), (1, 33, 128, 64, SEGMENTS), (3, 11, 128, 40, SEGMENTS), (1, 16, 128, 72, SEGMENTS),
    (1, 9, 128, 256, CHUNKS), (1, 34, 128, 64, CHUNKS), (1, 17, 128, 96, CHUNKS), (1, 37, 128, 32, CHUNKS), (2, 8, 128, 256, CHUNKS), (4, 8, 64, 128, CHUNKS),
    (5, 1, 64, 64, WALK), (1, 8, 192, 256, WALK), (1, 8, 60, 64, WALK), (1, 8, 64, 60, WALK)])
def test_segments_where_their_clusters_fit(seqs, heads, dim, vdim, want):
    f = pkg("_abi").lib().b200_debug_mlstm_route
    f.argtypes = [ctypes.c_int32] * 5
    assert f(seqs, heads, dim, vdim, 0) == want and f(seqs, heads, dim, vdim, 4000) == want


@pytest.mark.parametrize("seqs,dim,rows,want", [
    (1, 128, 1, WALK), (1, 128, 2, CHUNKS), (1, 128, 192, CHUNKS), (1, 128, 193, SEGMENTS), (2, 128, 2, WALK), (2, 128, 193, CHUNKS), (2, 128, 194, SEGMENTS),
    (1, 64, 256, CHUNKS), (1, 64, 257, SEGMENTS), (4, 40, 259, CHUNKS), (4, 40, 260, SEGMENTS), (4, 64, 4, WALK)])
def test_segments_where_a_portion_may_be_long_enough(seqs, dim, rows, want):
    f = pkg("_abi").lib().b200_debug_mlstm_route
    f.argtypes = [ctypes.c_int32] * 5
    assert f(seqs, 2, dim, 64, rows) == want
