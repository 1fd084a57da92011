"""Which kernels take a step of matrix memory: segments only where all of their clusters (of four CTAs, one an SM) run at a time."""
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
    f.argtypes = [ctypes.c_int32] * 4
    assert f(seqs, heads, dim, vdim) == want
