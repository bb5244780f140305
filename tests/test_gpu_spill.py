"""Pixel pairs shared over all warps (the spill pool) and the packed segment
walk: results against the oracle with every pair spilled after its first pixel
pair, at default, and with nothing spilled. Few vertices per pixel and many
(heavy pixel pairs are cut into shares), rings met by themselves (collinear
segments, shared vertices: the walk by sign codes), and coordinates beyond the
packed walk's range."""
import numpy as np
import pytest

from farm_gb300 import polygons as P
from farm_gb300.engine import Store
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _sets(seed, n_lo, n_hi, same):
    prm = P.StarParams(dom_hi=6.0, n_lo=n_lo, n_hi=n_hi)
    S = P.generate(prm, seed, 18)
    T = S if same else P.generate(prm, seed + 1, 30)
    return S, T, np.ascontiguousarray(P.mbr_join(S.mbrs(), T.mbrs()), np.uint32)


@pytest.mark.parametrize("budget", ["0", None, "1e30"])
@pytest.mark.parametrize("seed,n_lo,n_hi,vpr,same", [(71, 16, 60, 4, False), (72, 200, 3000, 10, False),
                                                     (73, 700, 2500, 700, False), (74, 16, 900, 10, True)])
def test_gpu_spilled_pairs_match_oracle(gpu_lib, monkeypatch, seed, n_lo, n_hi, vpr, same, budget):
    if budget is None:
        monkeypatch.delenv("FARM_SPILL_BUDGET", raising=False)
    else:
        monkeypatch.setenv("FARM_SPILL_BUDGET", budget)
    S, T, pairs = _sets(seed, n_lo, n_hi, same)
    RS, RT = O.rasterize_set(S, vpr), O.rasterize_set(T, vpr)
    with Store() as st:
        st.load_sets(S, T)
        st.rasterize(vpr=vpr)
        out, found = st.intersect(pairs)
        con, held = st.contain(pairs)
    exp = np.array([O.intersect(RS[s], RT[t]) for s, t in pairs], np.uint8)
    assert np.array_equal(out, exp), f"{int((out != exp).sum())} of {len(exp)} differ"
    assert found == int(exp.sum())
    exp = np.array([O.contain(RS[s], RT[t]) for s, t in pairs], np.uint8)
    assert np.array_equal(con, exp), f"{int((con != exp).sum())} of {len(exp)} differ"
    assert held == int(exp.sum())


@pytest.mark.parametrize("budget", ["0", None, "1e30"])
@pytest.mark.parametrize("seed,n_hi,vpr,geo,distance", [(81, 700, 10, False, 0.02), (82, 700, 4, False, 0.3),
                                                        (83, 1500, 700, False, 0.1), (84, 900, 10, True, 10.0),
                                                        (85, 300, 4, True, 150.0), (86, 200, 10, False, 1.5e5)])
def test_gpu_within_spilled_candidates_match_oracle(gpu_lib, monkeypatch, seed, n_hi, vpr, geo, distance, budget):
    if budget is None:
        monkeypatch.delenv("FARM_SPILL_BUDGET", raising=False)
    else:
        monkeypatch.setenv("FARM_SPILL_BUDGET", budget)
    prm = P.StarParams(dom_hi=9.0, n_hi=n_hi)
    S = P.generate(prm, seed, 40)
    pairs = np.array([(i, j) for i in range(40) for j in range(40) if i != j], np.uint32)
    RS = O.rasterize_set(S, vpr, True)
    with Store() as st:
        st.load_sets(S)
        st.rasterize(vpr=vpr, hierarchy=True)
        out, found = st.within(pairs, distance=distance, geography=geo, self_join=True)
        apx, _ = st.within(pairs, distance=distance, geography=geo, self_join=True, mode=1)
    exp = np.array([O.within(RS[s], RS[t], distance, geo) for s, t in pairs], np.uint8)
    assert np.array_equal(out, exp), f"{int((out != exp).sum())} of {len(exp)} differ"
    assert found == int(exp.sum())
    exp = np.array([O.within_heuristic(RS[s], RS[t], distance, geo) for s, t in pairs], np.uint8)
    assert np.array_equal(apx, exp), f"{int((apx != exp).sum())} of {len(exp)} differ (-a)"


@pytest.mark.parametrize("chunk", [1, 16, 32, 33])  # items of more than 32 edges are not cut
@pytest.mark.parametrize("seed,s_lo,s_hi,t_lo,t_hi,vpr", [(91, 8, 40, 9000, 14000, 10), (92, 600, 1500, 3000, 6000, 64),
                                                          (93, 2000, 3000, 2000, 3000, 10)])
def test_gpu_area_cut_items_match_oracle(gpu_lib, seed, s_lo, s_hi, t_lo, t_hi, vpr, chunk):
    S = P.generate(P.StarParams(dom_hi=2.0, r_lo=1.0, n_lo=s_lo, n_hi=s_hi), seed, 3)
    T = P.generate(P.StarParams(dom_hi=2.0, r_lo=1.0, n_lo=t_lo, n_hi=t_hi), seed + 1, 3)
    pairs = np.ascontiguousarray(P.mbr_join(S.mbrs(), T.mbrs()), np.uint32)
    assert len(pairs)
    with Store() as st:
        st.load_sets(S, T)
        st.rasterize(vpr=vpr)
        st.area_set_chunks([chunk] * 32)
        out = st.intersection_area(pairs)
        plan = st.area_plan(max_pairs=len(pairs), max_items=2 * 3 * (s_hi + t_hi) * 3)
        assert np.array_equal(plan.run(pairs), out)
        plan.close()
    for k, (s, t) in enumerate(pairs):
        exp = O.intersection_area(S.ring(s), T.ring(t))
        a = max(0.5 * abs(np.sum(r[:-1, 0] * r[1:, 1] - r[1:, 0] * r[:-1, 1]))
                for r in (S.ring(s).astype(np.float64), T.ring(t).astype(np.float64)))
        assert abs(out[k] - exp) <= 1e-9 * exp + 1e-14 * a, (k, s, t, out[k], exp)


@pytest.mark.parametrize("n", [1, 31, 33, 257, 20001])  # parts of a warp, of a block, several blocks
@pytest.mark.parametrize("n_lo,n_hi,vpr", [(8, 60, 4), (16, 4000, 10), (2000, 4000, 2000)])
def test_gpu_contain_points_flattened_match_oracle(gpu_lib, n_lo, n_hi, vpr, n):
    # pixels of a few edges to thousands, points on vertices, near them and anywhere
    S = P.generate(P.StarParams(dom_hi=3.0, n_lo=n_lo, n_hi=n_hi), 95, 7)
    rng = np.random.default_rng(n)
    pts = rng.uniform(-0.5, 3.5, (n, 2)).astype(np.float32)
    on = rng.integers(0, len(S.xy), n)
    pts = np.where((rng.random(n) < 0.5)[:, None], S.xy[on], pts).astype(np.float32)
    pairs = np.stack([rng.integers(0, 7, n), rng.permutation(n)], 1).astype(np.uint32)
    RS = O.rasterize_set(S, vpr)
    with Store() as st:
        st.load(0, S.off, S.xy)
        st.rasterize(vpr=vpr)
        out, found = st.contain_points(pts, pairs)
    exp = O.contain_points_many(RS, pts, pairs)
    assert np.array_equal(out, exp), f"{int((out != exp).sum())} of {n} differ"
    assert found == int(np.asarray(exp).sum())
