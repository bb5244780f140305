"""Device pair lists that start 4 bytes into an 8-byte word (a slice of an int32
tensor from an odd element on): every query reads them as any other list."""
import numpy as np
import pytest

from farm_gb300 import polygons as P
from farm_gb300.engine import MODE_APPROX, Store

pytestmark = pytest.mark.gpu


def test_gpu_pair_lists_at_odd_elements(gpu_lib):
    import torch

    prm = P.StarParams(dom_hi=6.0, r_lo=0.3, n_hi=500)
    S, T = P.generate(prm, 51, 40), P.generate(prm, 52, 60)
    pairs = np.ascontiguousarray(P.mbr_join(S.mbrs(), T.mbrs()), np.uint32)
    n = len(pairs)
    rng = np.random.default_rng(5)
    pts = rng.uniform(0, 6, (777, 2)).astype(np.float32)
    held = np.stack([rng.integers(0, S.n, 5003), rng.integers(0, 777, 5003)], 1).astype(np.uint32)

    def at(a, odd):
        buf = torch.zeros(a.size + 2, dtype=torch.int32, device="cuda:0")
        v = buf[int(odd):int(odd) + a.size].view(-1, 2)
        v.copy_(torch.from_numpy(a.view(np.int32)))
        assert v.data_ptr() % 8 == (4 if odd else 0)
        return v

    got = []
    with Store() as st:
        st.load_sets(S, T)
        st.rasterize(vpr=10, hierarchy=True)
        st.mlp_init(seed=3)
        plan = st.area_plan(max_pairs=n, max_items=100000)
        for odd in (False, True):
            d = at(pairs, odd)
            code, cost = st.filter_costs(d)
            got.append([st.intersect(d)[0], st.intersect(d, mode=MODE_APPROX)[0], st.contain(d)[0],
                        st.contain_points(torch.from_numpy(pts).cuda(), at(held, odd))[0],
                        st.within(d, distance=5.0)[0], st.intersection_area(d), plan.run(d), st.mlp_predict(d),
                        st.mlp_features(d)[:n].view(torch.int16), code, cost])
            got[-1] = [x.cpu().numpy() if hasattr(x, "cpu") else np.asarray(x) for x in got[-1]]
        plan.close()
    for a, b in zip(*got):
        assert len(a) and np.array_equal(a, b)
