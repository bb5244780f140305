"""Within between two polygons of one pixel each, whose sequences are their
whole rings: 46,342 points against 46,341 segments and back are more than 2^32
tests, so no count of them may be held in 32 bits. The rings come within the
distance at one spike only, past the target's first points."""
import numpy as np
import pytest

from farm_gb300 import polygons as P
from farm_gb300.engine import Store

pytestmark = pytest.mark.gpu

N = 46341  # edges; the ring in memory has one more vertex
AT = 50    # the vertex that faces the other ring
CELL = 1.1e-5 * 2 ** 17  # a step of the grid that rasters are aligned to


def _ring(col, facing, reach):
    """A circle in the middle of its cell, of 0.9 cells (its raster is that one pixel)."""
    a = facing + (np.arange(N) - AT) * (2 * np.pi / N)
    r = np.full(N, 0.45 * CELL)
    r[AT] = reach * CELL
    p = np.stack([(col + 0.5) * CELL + r * np.cos(a), 2.5 * CELL + r * np.sin(a)], 1)
    return np.concatenate([p, p[:1]])


def test_gpu_within_of_whole_rings_beyond_32_bit_counts(gpu_lib):
    assert 2 * (N + 1) * N > 2 ** 32
    # circles 0.1 cells apart; the second one's spike reaches to 0.055 cells from the first
    rings = [_ring(2, 0.0, 0.45), _ring(3, np.pi, 0.495)]
    off = np.array([0, N + 1, 2 * (N + 1)], np.uint64)
    pairs = np.array([[0, 1], [1, 0]], np.uint32)
    with Store() as st:
        st.load(0, off, np.ascontiguousarray(np.concatenate(rings), np.float32))
        st.rasterize(vpr=100000, hierarchy=True)
        for k in range(2):
            assert st.fetch_raster(0, k)["dimx"] * st.fetch_raster(0, k)["dimy"] == 1
        out, found = st.within(pairs, distance=0.08 * CELL, geography=False, self_join=True)
    assert out.tolist() == [1, 1] and found == 2
