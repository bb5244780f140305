"""A load that is refused (misaligned device vertices) or finds no memory for
its rings leaves the store as it was: the same number of polygons with other
offsets must not come to stand for the rings already loaded."""
import numpy as np
import pytest

from farm_gb300 import polygons as P
from farm_gb300.engine import Store

pytestmark = pytest.mark.gpu


def _no_memory(n):
    """n rings of 2^30 - 1 vertices: the ring array's allocation fails before a vertex is read."""
    return np.arange(n + 1, dtype=np.uint64) * (2 ** 30 - 1), np.zeros((1, 2), np.float32)


def _misaligned(n, total):
    """n rings of other lengths than the loaded ones', vertices 4 bytes into a device buffer."""
    import torch
    off = np.linspace(0, total, n + 1).astype(np.int64)
    buf = torch.zeros(2 * total + 1, dtype=torch.float32, device="cuda:0")
    return torch.from_numpy(off).cuda(), buf[1:].view(-1, 2)


@pytest.mark.parametrize("how", ["memory", "alignment"])
@pytest.mark.parametrize("side", [0, 1])
def test_gpu_failed_load_leaves_the_store_as_it_was(gpu_lib, how, side):
    prm = P.StarParams(dom_hi=20.0, n_hi=1200)
    S, T = P.generate(prm, 41, 400), P.generate(prm, 42, 400)
    with Store() as st:
        st.load_sets(S, T)
        st.rasterize(vpr=10)
        pairs = st.mbr_join()
        want, found = st.intersect(pairs)
        X = (S, T)[side]
        args = _no_memory(X.n) if how == "memory" else _misaligned(X.n, int(X.off[-1]))
        with pytest.raises(Exception, match="allocation" if how == "memory" else "8-byte"):
            st.load(side, *args)
        # the raster is still there, and made again it is the same
        for again in (False, True):
            if again:
                st.rasterize(vpr=10)
            assert np.array_equal(st.mbr_join(), pairs)
            out, f = st.intersect(pairs)
            assert np.array_equal(out, want) and f == found
        # and a proper load of that side goes through
        st.load(1, T.off, T.xy) if side else st.load_sets(S, T)
        st.rasterize(vpr=10)
        out, f = st.intersect(pairs)
        assert np.array_equal(out, want) and f == found
