"""The server's memory estimate of a request counts the slabs of the vertices
beside the buffers that grow with faces and positions."""
import ctypes

import pytest

from hostcheck import build as hb


@pytest.mark.parametrize("nfaces,nverts", [(2, 3), (1000, 502), (20_000, 60_000), (2_000, 3_000_000), (1 << 27, 1 << 26)])
def test_counts_vertex_slabs(nfaces, nverts):
    lib = ctypes.CDLL(hb._build("hc_footprint", "hostcheck_footprint.cpp"))
    lib.hc_footprint.restype = ctypes.c_int64
    got = lib.hc_footprint(ctypes.c_int64(nfaces), ctypes.c_int64(nverts))
    # per face, per vertex (positions), fixed, and 26 doubles per vertex with slabs: at most two a face have
    assert got >= 4096 * nfaces + 64 * nverts + (64 << 20) + 26 * 8 * min(nverts, 2 * nfaces)
